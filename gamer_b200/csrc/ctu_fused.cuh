// Hydro CTU as one plane-streaming kernel per patch group (PLM or PPM; five variables).
//
// Reference path replaced: CPU_FluidSolver_CTU without MHD
// (src/Model_Hydro/CPU_Hydro/CPU_FluidSolver_CTU.cpp:157-342, Hydro_TGradientCorrection :368-599).
//
// As separate kernels the stages exchange face states and fluxes through ~4.6 MB of global traffic per
// patch group (FP32), fifteen times the input and output.  Here one CTA sweeps a patch group along z
// and keeps every intermediate on chip.  A thread owns one column (i, j) of the 18 x 18 face-state
// cells; two phases per face-state plane k, each ended by one barrier:
//   (1) by columns: the z face states of plane k-1 corrected with the half-step x and y fluxes of that
//       plane, the full-step z flux between planes k-2 and k-1 and the output of plane k-2; then the
//       z reconstruction of plane k and the half-step z flux between planes k-1 and k, with which
//       the x and y face states of plane k-1 (in shared memory) are corrected; then the x and y
//       reconstruction of plane k;
//   (2) by faces: the half-step x and y Riemann problems of plane k and the full-step ones of plane
//       k-1, and the conversion of an input plane to primitive variables.
// Everything along z (uncorrected and corrected face states, half- and full-step fluxes) is private to
// the column's thread.  Input planes arrive by 1-D bulk copies into a ring, the next patch group's
// first planes during the last steps of the current one.
// FP32 PLM HLLC: 107 KB of shared memory and 80 registers (48 bytes spilled), two CTAs of 352 threads per SM.
// Bound by the barriers between the phases and by dependent instructions, at 56% of the issue slots.
#pragma once
#include "ctu_hydro.cuh"
#include "hydro_pair.cuh"
#include "tma.cuh"

namespace gb {
namespace hctu {

constexpr int FU_THREADS = 352;                    // 18 x 18 columns in whole warps
constexpr int FU_CELLS = NF*NF;                    // face-state cells of a plane
constexpr int FU_HALF = ( NF - 1 )*NF;             // half-step x (and y) faces of a plane
constexpr int FU_FULL = ( NF - 1 )*PS2;            // full-step x (and y) faces of a plane

// shared memory (bytes): mbarriers, the ring of input planes, the x and y face states of two planes,
// the half- and the full-step x and y fluxes of one plane
template <typename R, int NC, int LR> struct FusedSmem {
   static constexpr int LIVE = 2*G<LR>::LRG + 1;   // input planes that one reconstruction reads
   static constexpr int NSLOT = LIVE + 1;
   static constexpr int PLANE = NC*G<LR>::NX*G<LR>::NX;
   static constexpr int o_ring = 128;
   static constexpr int o_fc = o_ring + NSLOT*PLANE*(int)sizeof(R);          // [2 planes][x, y][2 sides][NC][18*18]
   static constexpr int o_fh = o_fc + 2*2*2*NC*FU_CELLS*(int)sizeof(R);      // [x, y][NC][306]
   static constexpr int o_ff = o_fh + 2*NC*FU_HALF*(int)sizeof(R);           // [x, y][NC][272]
   static constexpr int bytes = o_ff + 2*NC*FU_FULL*(int)sizeof(R);
};

// the two faces of a cell along one direction, primitive -> conserved (pri2con on both lanes)
template <int NC>
GB_DEV void faces_con( const Phys<float> &ph, const float (&fl)[NC], const float (&fr)[NC], float2 (&u)[NC] )
{
   float2 w[NC];
#  pragma unroll
   for (int v=0; v<NC; v++) w[v] = make_float2( fl[v], fr[v] );
   u[0] = w[0];
   u[1] = p_mul( w[0], w[1] );
   u[2] = p_mul( w[0], w[2] );
   u[3] = p_mul( w[0], w[3] );
   float2 v2 = p_mul( w[1], w[1] );
   v2 = p_fma( w[2], w[2], v2 );
   v2 = p_fma( w[3], w[3], v2 );
   u[4] = p_fma( w[4], p_bc( ph.inv_gm1 ), p_mul( p_mul( p_bc( 0.5f ), w[0] ), v2 ) );
}
template <int NC>
GB_DEV void faces_con( const Phys<double> &ph, const double (&fl)[NC], const double (&fr)[NC], double2 (&u)[NC] )
{
   double l[NC], r[NC];
   pri2con<NC>( ph, fl, l );
   pri2con<NC>( ph, fr, r );
#  pragma unroll
   for (int v=0; v<NC; v++) u[v] = make_double2( l[v], r[v] );
}

// the transverse-gradient correction c of both faces, density and internal-energy floors
template <int P, int NC>
GB_DEV void faces_correct( const Phys<float> &ph, const float (&c)[NC], float2 (&q)[NC] )
{
#  pragma unroll
   for (int v=0; v<NC; v++) q[v] = p_add( q[v], p_bc( c[v] ) );
   q[0] = make_float2( fmaxf( q[0].x, ph.min_dens ), fmaxf( q[0].y, ph.min_dens ) );
   q[4] = floor_eint_pair<P>( ph, q[0], q[1], q[2], q[3], q[4] );
}
template <int P, int NC>
GB_DEV void faces_correct( const Phys<double> &ph, const double (&c)[NC], double2 (&q)[NC] )
{
#  pragma unroll
   for (int v=0; v<NC; v++) { q[v].x += c[v];  q[v].y += c[v]; }
   q[0].x = gmax( q[0].x, ph.min_dens );  q[0].y = gmax( q[0].y, ph.min_dens );
   q[4].x = floor_eint_in_engy<P>( ph, q[0].x, q[1].x, q[2].x, q[3].x, q[4].x );
   q[4].y = floor_eint_in_engy<P>( ph, q[0].y, q[1].y, q[2].y, q[3].y, q[4].y );
}

template <typename R> struct TwoOf;
template <> struct TwoOf<float>  { typedef float2 type; };
template <> struct TwoOf<double> { typedef double2 type; };

// GMM: generalized MinMod with theta < 2 built in (its PLM clamps never act); otherwise the run-time
// limiter
template <typename R, int P, int RS, int NC, int LR, bool GMM>
__global__ void __launch_bounds__( FU_THREADS, ( sizeof(R) == 4 && LR == LR_PLM ) ? 2 : 1 )
hctu_fused_kernel( const __grid_constant__ Args<R> a, int *status )
{
   typedef FusedSmem<R,NC,LR> S;
   typedef typename TwoOf<R>::type R2;
   typedef typename std::conditional<P == P_MIXED, double, R>::type A;   // accumulation type
   constexpr int N = G<LR>::NX, N2 = N*N, LRG = G<LR>::LRG, FLG = G<LR>::FLG;
   constexpr int LIVE = S::LIVE, NSLOT = S::NSLOT, PLANE = S::PLANE;
   constexpr bool X2 = std::is_same<R, float>::value && RS == RS_HLLC && NC == 5;
   static_assert( NC == 5, "five variables" );
   extern __shared__ __align__(128) unsigned char smem[];
   uint64_t *bar = (uint64_t*)smem;                 // one mbarrier per ring slot
   int *s_abort  = (int*)( smem + 64 );
   R *s_ring = (R*)( smem + S::o_ring );
   R *s_fc   = (R*)( smem + S::o_fc );
   R *s_fh   = (R*)( smem + S::o_fh );
   R *s_ff   = (R*)( smem + S::o_ff );
   const int tid = threadIdx.x, nth = FU_THREADS;
   const Phys<R> ph = a.ph;
   const int lim = GMM ? LIM_GMINMOD : a.limiter;
   const bool clamp = GMM ? false : plm_clamp_needed( lim, (double)a.coeff );
   const R dt_dh2 = R(0.5)*a.dt/a.dh;
   const A dt_dh  = (A)a.dt/(A)a.dh;

   if ( tid == 0 )
   {
      for (int q=0; q<NSLOT; q++) mbar_init( &bar[q], 1 );
      mbar_init_fence();
      *s_abort = 0;
   }
   __syncthreads();

   // the planes of this CTA's patch groups as one sequence: plane s is input plane s % N of its
   // (s / N)-th patch group, in ring slot s % NSLOT
   const int npg_cta = ( a.npg - (int)blockIdx.x + (int)gridDim.x - 1 )/(int)gridDim.x;
   const int nplane = npg_cta*N;
   auto issue = [&]( int s ) {
      if ( s >= nplane ) return;
      const int q = s % NSLOT, c = s % N;
      const R *g = a.in + (size_t)( blockIdx.x + (size_t)( s/N )*gridDim.x )*NC*N*N2 + (size_t)c*N2;
      fence_proxy_async();
      mbar_expect_tx( &bar[q], PLANE*sizeof(R) );
      for (int v=0; v<NC; v++) bulk_g2s( s_ring + ( q*NC + v )*N2, g + (size_t)v*N*N2, N2*sizeof(R), &bar[q] );
   };
   // wait for plane s and convert it in place; the calling thread is number vt of the CTA's
   auto convert = [&]( int s, int vt ) {
      if ( s >= nplane ) return;
      if ( !mbar_wait_bounded( &bar[s % NSLOT], ( s/NSLOT ) & 1 ) )
      {
         atomicOr( status, GB_ST_TMA_TIMEOUT );
         *s_abort = 1;
      }
      R *pt = s_ring + ( s % NSLOT )*PLANE;
      if constexpr ( std::is_same<R, float>::value )
      {
         for (int e = vt; e < N2/2; e += nth)
         {
            float2 u[NC], w[NC];
#           pragma unroll
            for (int v=0; v<NC; v++) u[v] = ( (float2*)( pt + v*N2 ) )[e];
            con2pri_cc_pair<P,NC>( ph, u, w );
#           pragma unroll
            for (int v=0; v<NC; v++) ( (float2*)( pt + v*N2 ) )[e] = w[v];
         }
      }
      else
      {
         for (int e = vt; e < N2; e += nth)
         {
            R u[NC], w[NC];
#           pragma unroll
            for (int v=0; v<NC; v++) u[v] = pt[v*N2 + e];
            con2pri_cc<P,NC>( ph, u, w );
#           pragma unroll
            for (int v=0; v<NC; v++) pt[v*N2 + e] = w[v];
         }
      }
   };
   // a copy never arrived: wait once more (bounded) for the copies that may be in flight, then give up
   auto bail = [&]( int s0, int s1 ) {
      if ( tid == 0 )
         for (int s = s0; s <= s1 && s < nplane; s++) mbar_wait_bounded( &bar[s % NSLOT], ( s/NSLOT ) & 1 );
      __syncthreads();
   };

   // the column of this thread: the inner 16 x 16 first, then the ring around it
   int i, j;
   const bool col = ( tid < FU_CELLS ), inner = ( tid < PS2*PS2 );
   if ( inner ) { i = 1 + tid % PS2;  j = 1 + tid / PS2; }
   else
   {
      const int h = tid - PS2*PS2;
      if      ( h < NF )          { i = h;             j = 0;      }
      else if ( h < 2*NF )        { i = h - NF;        j = NF - 1; }
      else if ( h < 2*NF + PS2 )  { i = 0;             j = 1 + h - 2*NF; }
      else                        { i = NF - 1;        j = ( 1 + h - 2*NF - PS2 < NF ) ? 1 + h - 2*NF - PS2 : NF - 1; }
   }
   const bool in_i = ( i >= 1 && i <= PS2 ), in_j = ( j >= 1 && j <= PS2 );
   const int f = j*NF + i, cell = ( j + LRG )*N + i + LRG;

   if ( tid == 0 ) for (int s=0; s<=LIVE; s++) issue( s );
   for (int s=0; s<LIVE; s++) convert( s, tid );
   __syncthreads();
   if ( *s_abort ) { bail( 0, LIVE );  return; }

   for (int t=0; t<npg_cta; t++)
   {
      const size_t pg = blockIdx.x + (size_t)t*gridDim.x;
      const int s0 = t*N;                            // sequence number of this patch group's plane 0
      const R *g_in = a.in + pg*NC*N*N2;
      R *g_out  = a.out + pg*NC*PS2*PS2*PS2;
      R *g_flux = ( a.flux != nullptr ) ? a.flux + pg*9*NC*PS2*PS2 : nullptr;
      // carried from plane to plane: the uncorrected z faces of plane k-1 (x = lower, y = upper), the
      // corrected upper z face of plane k-2, the half-step z flux below plane k-1 and the full-step
      // z flux below plane k-2
      R2 zf[NC];
      R czu[NC], fzh[NC], fzf[NC];
#     pragma unroll
      for (int v=0; v<NC; v++) { zf[v].x = zf[v].y = R(0);  czu[v] = fzh[v] = fzf[v] = R(0); }

      for (int k=0; k<=NF; k++)
      {
         if ( col )
         {
            // half-step transverse flux differences of plane k-1 at this column
            auto dfx = [&]( int v ) { const R *F = s_fh + v*FU_HALF + j*( NF - 1 ) + i;  return F[0] - F[-1]; };
            auto dfy = [&]( int v ) { const R *F = s_fh + ( NC + v )*FU_HALF + j*NF + i;  return F[0] - F[-NF]; };
            if ( k >= 1 && inner )
            {
               R2 q[NC];
               R c[NC];
#              pragma unroll
               for (int v=0; v<NC; v++) { q[v] = zf[v];  c[v] = -dt_dh2*( dfx( v ) + dfy( v ) ); }
               faces_correct<P,NC>( ph, c, q );
               if ( k >= 2 )
               {
                  R L[NC], Rr[NC], F[NC];
#                 pragma unroll
                  for (int v=0; v<NC; v++) { L[v] = czu[v];  Rr[v] = q[v].x; }
                  riemann<RS,2,P,NC>( ph, L, Rr, F );
                  const int ko = k - 2;
                  if ( g_flux != nullptr && ( ko & 7 ) == 0 )
                  {
                     R *dst = g_flux + (size_t)( ( 6 + ( ko >> 3 ) )*NC )*PS2*PS2 + tid;
#                    pragma unroll
                     for (int v=0; v<NC; v++) dst[v*PS2*PS2] = F[v];
                  }
                  if ( k >= 3 )
                  {
                     // output plane o = k-3 is face-state plane k-2 (Hydro_FullStepUpdate,
                     // CPU_Shared_FullStepUpdate.cpp:64-140)
                     const int o = k - 3, oi = i - 1, oj = j - 1;
                     const R *u = g_in + (size_t)( o + FLG )*N2 + ( oj + FLG )*N + oi + FLG;
#                    pragma unroll
                     for (int v=0; v<NC; v++)
                     {
                        const R *fx = s_ff + v*FU_FULL + oj*( NF - 1 ) + oi, *fy = s_ff + ( NC + v )*FU_FULL + oj*PS2 + oi;
                        const A dx = (A)fx[1] - (A)fx[0], dy = (A)fy[PS2] - (A)fy[0], dz = (A)F[v] - (A)fzf[v];
                        g_out[v*PS2*PS2*PS2 + o*PS2*PS2 + tid] = (R)( (A)u[(size_t)v*N*N2] - dt_dh*( ( dx + dy ) + dz ) );
                     }
                  }
#                 pragma unroll
                  for (int v=0; v<NC; v++) fzf[v] = F[v];
               }
#              pragma unroll
               for (int v=0; v<NC; v++) czu[v] = q[v].y;
            }
            if ( k < NF )
            {
               const R *pc = s_ring + ( ( s0 + k + LRG ) % NSLOT )*PLANE + cell;
               R cc[NC];
#              pragma unroll
               for (int v=0; v<NC; v++) cc[v] = pc[v*N2];
               R fl[NC], fr[NC];
               {
                  const R *pl = s_ring + ( ( s0 + k + LRG - 1 ) % NSLOT )*PLANE + cell;
                  const R *pr = s_ring + ( ( s0 + k + LRG + 1 ) % NSLOT )*PLANE + cell;
                  const R *pll = ( LR == LR_PPM ) ? s_ring + ( ( s0 + k ) % NSLOT )*PLANE + cell : nullptr;
                  const R *prr = ( LR == LR_PPM ) ? s_ring + ( ( s0 + k + 2*LRG ) % NSLOT )*PLANE + cell : nullptr;
                  hctu_faces<2,RS,NC,0,LR>( ph, lim, a.coeff, clamp, dt_dh2, pll, pl, cc, pr, prr, N2, fl, fr );
               }
               R2 z[NC];
               faces_con( ph, fl, fr, z );
               if ( k >= 1 && ( in_i || in_j ) )
               {
                  R L[NC], Rr[NC], F[NC];
#                 pragma unroll
                  for (int v=0; v<NC; v++) { L[v] = zf[v].y;  Rr[v] = z[v].x; }
                  riemann<RS,2,P,NC>( ph, L, Rr, F );
                  if ( k >= 2 )
                  {
                     // the x and y face states of plane k-1, corrected in place
                     R *sx = s_fc + ( ( k - 1 ) & 1 )*4*NC*FU_CELLS + f, *sy = sx + 2*NC*FU_CELLS;
                     R2 q[NC];
                     R c[NC];
                     if ( in_j )
                     {
#                       pragma unroll
                        for (int v=0; v<NC; v++)
                        {
                           q[v].x = sx[v*FU_CELLS];  q[v].y = sx[( NC + v )*FU_CELLS];
                           c[v] = -dt_dh2*( dfy( v ) + ( F[v] - fzh[v] ) );
                        }
                        faces_correct<P,NC>( ph, c, q );
#                       pragma unroll
                        for (int v=0; v<NC; v++) { sx[v*FU_CELLS] = q[v].x;  sx[( NC + v )*FU_CELLS] = q[v].y; }
                     }
                     if ( in_i )
                     {
#                       pragma unroll
                        for (int v=0; v<NC; v++)
                        {
                           q[v].x = sy[v*FU_CELLS];  q[v].y = sy[( NC + v )*FU_CELLS];
                           c[v] = -dt_dh2*( ( F[v] - fzh[v] ) + dfx( v ) );
                        }
                        faces_correct<P,NC>( ph, c, q );
#                       pragma unroll
                        for (int v=0; v<NC; v++) { sy[v*FU_CELLS] = q[v].x;  sy[( NC + v )*FU_CELLS] = q[v].y; }
                     }
                  }
#                 pragma unroll
                  for (int v=0; v<NC; v++) fzh[v] = F[v];
               }
#              pragma unroll
               for (int v=0; v<NC; v++) zf[v] = z[v];
               // x and y face states of plane k
               R *sx = s_fc + ( k & 1 )*4*NC*FU_CELLS + f, *sy = sx + 2*NC*FU_CELLS;
               R2 u[NC];
               hctu_faces<0,RS,NC,0,LR>( ph, lim, a.coeff, clamp, dt_dh2, pc - 2, pc - 1, cc, pc + 1, pc + 2, N2, fl, fr );
               faces_con( ph, fl, fr, u );
#              pragma unroll
               for (int v=0; v<NC; v++) { sx[v*FU_CELLS] = u[v].x;  sx[( NC + v )*FU_CELLS] = u[v].y; }
               hctu_faces<1,RS,NC,0,LR>( ph, lim, a.coeff, clamp, dt_dh2, pc - 2*N, pc - N, cc, pc + N, pc + 2*N, N2, fl, fr );
               faces_con( ph, fl, fr, u );
#              pragma unroll
               for (int v=0; v<NC; v++) { sy[v*FU_CELLS] = u[v].x;  sy[( NC + v )*FU_CELLS] = u[v].y; }
            }
         }
         __syncthreads();
         // the slot of the oldest plane of this reconstruction is free; the last step frees the others
         if ( tid == 0 )
         {
            if ( k < NF ) issue( s0 + k + NSLOT );
            else for (int q=2; q<=LIVE; q++) issue( s0 + N + q );
         }
         int nitem = 0;
         if ( k < NF )
         {
            const bool full = ( k >= 2 );             // plane k-1 in 1..16
            nitem = FU_HALF + ( full ? FU_FULL : 0 );
            if constexpr ( X2 )
            {
               // x face e and y face e of one kind as the two lanes of one HLLC, rotated frame
               constexpr int ry[5] = { 0, 2, 3, 1, 4 };
               for (int e = tid; e < nitem; e += nth)
               {
                  const bool fs = ( e >= FU_HALF );
                  const int e2 = fs ? e - FU_HALF : e;
                  const int ix = e2 % ( NF - 1 ), jx = e2 / ( NF - 1 ) + ( fs ? 1 : 0 );
                  const int iy = fs ? 1 + e2 % PS2 : e2 % NF, jy = fs ? e2 / PS2 : e2 / NF;
                  const R *sx = s_fc + ( ( fs ? k - 1 : k ) & 1 )*4*NC*FU_CELLS, *sy = sx + 2*NC*FU_CELLS;
                  const int ox = jx*NF + ix, oy = jy*NF + iy;
                  float2 L[5], Rr[5], F[5];
#                 pragma unroll
                  for (int q=0; q<5; q++)
                  {
                     L[q]  = make_float2( sx[( NC + q )*FU_CELLS + ox], sy[( NC + ry[q] )*FU_CELLS + oy] );
                     Rr[q] = make_float2( sx[q*FU_CELLS + ox + 1],      sy[ry[q]*FU_CELLS + oy + NF] );
                  }
                  bool nan_x, nan_y;
                  riemann_hllc_x2<P>( ph, L, Rr, F, nan_x, nan_y );
                  float Fx[5], Fy[5];
#                 pragma unroll
                  for (int q=0; q<5; q++) { Fx[q] = F[q].x;  Fy[ry[q]] = F[q].y; }
                  if ( nan_x || nan_y )
                  {
                     // HLLE rescue of a NaN flux (CPU_Shared_ComputeFlux.cpp:313-362), per face
                     float l[5], r[5];
                     if ( nan_x )
                     {
#                       pragma unroll
                        for (int q=0; q<5; q++) { l[q] = L[q].x;  r[q] = Rr[q].x; }
                        riemann_hlle_outlined<0,P,5>( ph, l, r, Fx );
                     }
                     if ( nan_y )
                     {
#                       pragma unroll
                        for (int q=0; q<5; q++) { l[ry[q]] = L[q].y;  r[ry[q]] = Rr[q].y; }
                        riemann_hlle_outlined<1,P,5>( ph, l, r, Fy );
                     }
                  }
                  R *dx = fs ? s_ff + e2 : s_fh + e2;
                  const int st = fs ? FU_FULL : FU_HALF;
#                 pragma unroll
                  for (int v=0; v<NC; v++) { dx[v*st] = Fx[v];  dx[( NC + v )*st] = Fy[v]; }
                  if ( fs && g_flux != nullptr )
                  {
                     const int ko = k - 2;
                     if ( ( ix & 7 ) == 0 )
                     {
                        R *dst = g_flux + (size_t)( ( ix >> 3 )*NC )*PS2*PS2 + ko*PS2 + jx - 1;
#                       pragma unroll
                        for (int v=0; v<NC; v++) dst[v*PS2*PS2] = Fx[v];
                     }
                     if ( ( jy & 7 ) == 0 )
                     {
                        R *dst = g_flux + (size_t)( ( 3 + ( jy >> 3 ) )*NC )*PS2*PS2 + ko*PS2 + iy - 1;
#                       pragma unroll
                        for (int v=0; v<NC; v++) dst[v*PS2*PS2] = Fy[v];
                     }
                  }
               }
            }
            else
            {
               nitem *= 2;
               for (int e = tid; e < nitem; e += nth)
               {
                  const bool fs = ( e >= 2*FU_HALF );
                  const int nf = fs ? FU_FULL : FU_HALF;
                  const int e1 = fs ? e - 2*FU_HALF : e;
                  const bool ydir = ( e1 >= nf );
                  const int e2 = ydir ? e1 - nf : e1, wx = fs ? PS2 : NF, o = fs ? 1 : 0;
                  const R *sd = s_fc + ( ( fs ? k - 1 : k ) & 1 )*4*NC*FU_CELLS + ( ydir ? 2*NC*FU_CELLS : 0 );
                  const int fi = ydir ? o + e2 % wx : e2 % ( NF - 1 ), fj = ydir ? e2 / wx : o + e2 / ( NF - 1 );
                  const R *pl = sd + NC*FU_CELLS + fj*NF + fi, *pr = sd + fj*NF + fi + ( ydir ? NF : 1 );
                  R L[NC], Rr[NC], F[NC];
#                 pragma unroll
                  for (int v=0; v<NC; v++) { L[v] = pl[v*FU_CELLS];  Rr[v] = pr[v*FU_CELLS]; }
                  if ( ydir ) riemann<RS,1,P,NC>( ph, L, Rr, F );
                  else        riemann<RS,0,P,NC>( ph, L, Rr, F );
                  R *d = ( fs ? s_ff : s_fh ) + ( ydir ? NC*nf : 0 ) + e2;
#                 pragma unroll
                  for (int v=0; v<NC; v++) d[v*nf] = F[v];
                  if ( fs && g_flux != nullptr )
                  {
                     const int nrm = ydir ? fj : fi, tr = ( ydir ? fi : fj ) - 1;
                     if ( ( nrm & 7 ) == 0 )
                     {
                        R *dst = g_flux + (size_t)( ( ( ydir ? 3 : 0 ) + ( nrm >> 3 ) )*NC )*PS2*PS2 + ( k - 2 )*PS2 + tr;
#                       pragma unroll
                        for (int v=0; v<NC; v++) dst[v*PS2*PS2] = F[v];
                     }
                  }
               }
            }
            // the next plane of this patch group, dealt out from the first thread with one item fewer
            if ( k + LIVE < N ) convert( s0 + k + LIVE, ( tid + nth - nitem % nth ) % nth );
         }
         else for (int q=0; q<LIVE; q++) convert( s0 + N + q, tid );
         __syncthreads();
         if ( *s_abort ) { bail( s0 + k + LIVE, ( k < NF ) ? s0 + k + NSLOT : s0 + N + LIVE );  return; }
      }
   }
}

} // namespace hctu

// one launch over all npg patch groups (persistent grid, no scratch)
template <typename R, int P, int RS, int LR, bool GMM>
cudaError_t hctu_fused_launch( const hctu::Args<R> &a, int *status, cudaStream_t st )
{
   using namespace hctu;
   const void *fn = (const void*)hctu_fused_kernel<R,P,RS,5,LR,GMM>;
   constexpr int smem = FusedSmem<R,5,LR>::bytes;
   int dev = 0, nsm = 0, per_sm = 0;
   cudaGetDevice( &dev );
   cudaDeviceGetAttribute( &nsm, cudaDevAttrMultiProcessorCount, dev );
   cudaError_t e = cudaFuncSetAttribute( fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem );
   if ( e == cudaSuccess ) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor( &per_sm, fn, FU_THREADS, smem );
   if ( e != cudaSuccess ) return e;
   if ( per_sm < 1 ) return cudaErrorInvalidConfiguration;
   const int grid = ( nsm*per_sm < a.npg ) ? nsm*per_sm : a.npg;
   hctu_fused_kernel<R,P,RS,5,LR,GMM><<< grid, FU_THREADS, smem, st >>>( a, status );
   return cudaGetLastError();
}

// a call of one precision policy: the solvers, reconstructions and limiter kinds that ctu_hydro_fused has a
// line for
template <typename R, int P, int RS, int LR>
int hctu_fused_call( const gb_fluid_config &cfg, const void *in, void *out, void *flux, int npg, const gb_fluid_params *prm,
                     int *status, cudaStream_t st )
{
   const hctu::Args<R> a = hctu_args<R,5,LR>( cfg, in, out, flux, nullptr, 0, npg, prm );
   if ( hctu_gmm( *prm ) ) return ( hctu_fused_launch<R,P,RS,LR,true>( a, status, st ) == cudaSuccess ) ? GB_OK : GB_E_CUDA;
   if constexpr ( P != P_MIXED && !( LR == LR_PPM && RS == RS_HLLE ) )
      return ( hctu_fused_launch<R,P,RS,LR,false>( a, status, st ) == cudaSuccess ) ? GB_OK : GB_E_CUDA;
   return GB_E_UNSUPPORTED;
}

template <typename R, int P>
int hctu_fused_pick( const gb_fluid_config &cfg, const void *in, void *out, void *flux, int npg, const gb_fluid_params *prm,
                     int *status, cudaStream_t st )
{
   if ( cfg.rsolver != GB_RSOLVER_HLLC && cfg.rsolver != GB_RSOLVER_HLLE ) return GB_E_UNSUPPORTED;
   const bool hlle = ( cfg.rsolver == GB_RSOLVER_HLLE );
   if ( cfg.lr_scheme == GB_LR_PPM )
   {
      if constexpr ( P == P_FP32 )
         return hlle ? hctu_fused_call<R,P,RS_HLLE,LR_PPM>( cfg, in, out, flux, npg, prm, status, st )
                     : hctu_fused_call<R,P,RS_HLLC,LR_PPM>( cfg, in, out, flux, npg, prm, status, st );
      else
         return GB_E_UNSUPPORTED;
   }
   return hlle ? hctu_fused_call<R,P,RS_HLLE,LR_PLM>( cfg, in, out, flux, npg, prm, status, st )
               : hctu_fused_call<R,P,RS_HLLC,LR_PLM>( cfg, in, out, flux, npg, prm, status, st );
}

} // namespace gb
