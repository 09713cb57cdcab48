// The adjoint step of adjoint.cuh as one plane-streaming kernel per patch group (float, HLLC).
//
// As separate kernels the stages exchange the face states, the tape, the face adjoints (double) and the
// cell adjoints (double, added atomically) through ~10 MB of global traffic per patch group, after
// clearing ~2 MB of it.  Here one CTA sweeps a patch group along z; a thread owns one column (i, j) of
// the 18 x 18 face-state cells.  Two phases per face-state plane k, each ended by one barrier:
//   (1) by columns: the face states of plane k; the adjoint of the z Riemann problem between planes
//       k-1 and k; the cell adjoint of plane k-1 (Hancock, limiter), whose parts for the neighbours
//       in the plane go to shared memory and those along z stay with the column; then the cells of
//       input plane k-1 are complete, and their gradient is written;
//   (2) by faces: the adjoints of the x and y Riemann problems of plane k; each column adds its
//       neighbours' parts of plane k-1, the cells around the 18 x 18 columns are written, and an
//       input plane is converted to primitive variables.
// Every adjoint is added by the thread that owns it, in a fixed order (no atomics, nothing to clear).
// Sums are in double as in the separate kernels.  The planes of the input (ring of 5) and of
// d loss / d U_out (ring of 4) arrive by 1-D bulk copies; 213 KB of shared memory, one CTA of 384
// threads per SM at 162 registers.  The global traffic per patch group is the input, d loss / d U_out and
// d loss / d U_in, 0.5 MB.  Bound by the barriers between the phases and by dependent instructions, with three
// warps per scheduler to hide them (42% of the issue slots), which is what a wave costs whatever it
// holds: a wave of 148 patch groups takes 0.227 ms where the separate kernels take 0.33; 1024 patch
// groups, two steps forward and back: 2.28 -> 1.71 ms a step.
#pragma once
#include "adjoint.cuh"
#include "hydro_pair.cuh"
#include "tma.cuh"

namespace gb {

constexpr int AF_THREADS = 384;
constexpr int AF_CELLS = ADJ_F*ADJ_F, AF_FACES = NFLX*PS2;        // columns; x (and y) faces of a plane
constexpr int AF_N2 = ADJ_N*ADJ_N, AF_PLANE = ADJ_NC*AF_N2, AF_SLOTS = 5, AF_GSLOTS = 4;
constexpr int AF_BORDER = 4*( ADJ_N - 1 );                        // input cells of a plane around the columns

struct AdjFusedSmem {
   static constexpr int o_ring = 128;
   static constexpr int o_fc = o_ring + AF_SLOTS*AF_PLANE*4;      // [x, y][2 sides][5][18*18] face states (float)
   static constexpr int o_q  = o_fc + 2*2*ADJ_NC*AF_CELLS*4;      // [x, y][2 cells][5][272] face adjoints (double)
   static constexpr int o_c  = o_q + 2*2*ADJ_NC*AF_FACES*8;       // [x-, x+, y-, y+][5][18*18] parts for the neighbours (double)
   static constexpr int o_g  = o_c + 4*ADJ_NC*AF_CELLS*8;         // ring of 4 planes [5][16*16] of d loss / d U_out (double)
   static constexpr int o_z  = o_g + AF_GSLOTS*ADJ_NC*PS2*PS2*8;  // zeros in the place of the adjoints of absent faces (double)
   static constexpr int bytes = o_z + ADJ_NC*AF_FACES*8;
};

// a face whose HLLC flux is NaN (the HLLE rescue applies): forward-mode dual numbers, out of line and
// by value, so that the states of the ordinary faces stay in registers
struct AdjFaceIn  { float l[ADJ_NC], r[ADJ_NC];  double f[ADJ_NC]; };
struct AdjFaceOut { double l[ADJ_NC], r[ADJ_NC]; };

template <int D, int P>
__device__ __noinline__ AdjFaceOut adj_face_dual_rare( const Phys<float> ph, const AdjFaceIn x )
{
   typedef Dual<ADJ_NC,float> DR;
   const Phys<DR> dph = dual_phys<float,ADJ_NC>( ph );
   AdjFaceOut o;
   for (int side=0; side<2; side++)
   {
      DR dl[ADJ_NC], dr[ADJ_NC], fo[ADJ_NC];
#     pragma unroll
      for (int v=0; v<ADJ_NC; v++)
      {
         dl[v] = side ? DR( (double)x.l[v] ) : DR::var( x.l[v], v );
         dr[v] = side ? DR::var( x.r[v], v ) : DR( (double)x.r[v] );
      }
      riemann<RS_HLLC,D,P,ADJ_NC>( dph, dl, dr, fo );
#     pragma unroll
      for (int w=0; w<ADJ_NC; w++)
      {
         double s = 0.0;
#        pragma unroll
         for (int v=0; v<ADJ_NC; v++) s += x.f[v]*(double)fo[v].d[w];
         if ( side ) o.r[w] = s; else o.l[w] = s;
      }
   }
   return o;
}

// the adjoints lb, rb of the face states ql, qr from that of their HLLC flux; a NaN flux is reported in *nan
// (RESCUE: differentiated as the HLLE rescue)
template <int D, int P, bool RESCUE>
GB_DEV void adj_face_hllc( const Phys<float> &ph, const float (&ql)[ADJ_NC], const float (&qr)[ADJ_NC], const double (&fbar)[ADJ_NC],
                           double (&lb)[ADJ_NC], double (&rb)[ADJ_NC], int *nan )
{
   if ( hllc_vjp<D,float>( ph, ql, qr, fbar, lb, rb ) ) return;
   if constexpr ( !RESCUE )
   {
      *nan = 1;
#     pragma unroll
      for (int v=0; v<ADJ_NC; v++) lb[v] = rb[v] = 0.0;
      return;
   }
   AdjFaceIn x;
#  pragma unroll
   for (int v=0; v<ADJ_NC; v++) { x.l[v] = ql[v];  x.r[v] = qr[v];  x.f[v] = fbar[v]; }
   const AdjFaceOut o = adj_face_dual_rare<D,P>( ph, x );
#  pragma unroll
   for (int v=0; v<ADJ_NC; v++) { lb[v] = o.l[v];  rb[v] = o.r[v]; }
}

// d loss / d U_in of one input cell: J_Con2Pri^T wb from its primitive variables w (stride AF_N2), the
// reset part (ext: already in gin) and the identity term of an output cell (g, or null)
template <int P>
GB_DEV void adj_cell_out( const AdjArgs<float> &a, size_t pg, int c, const double (&wb)[ADJ_NC], const float *w, bool ext,
                          const double *g )
{
   double *gi = a.gin + pg*ADJ_NC*ADJ_N3 + c;
   double out[ADJ_NC];
   bool any = false;
#  pragma unroll
   for (int v=0; v<ADJ_NC; v++) { any |= ( wb[v] != 0.0 );  out[v] = 0.0; }
   if ( ext )
   {
#     pragma unroll
      for (int v=0; v<ADJ_NC; v++) out[v] = gi[v*ADJ_N3];
   }
   if ( any )
   {
      const float pr = w[4*AF_N2];
      bool floored = false;
      if ( pr == a.ph.min_pres )
      {
         // the floor passes nothing on: whether it acted shows in the unfloored pressure
         const float *u = a.in + pg*ADJ_NC*ADJ_N3 + c;
         const float d = u[0], m1 = u[ADJ_N3], m2 = u[2*ADJ_N3], m3 = u[3*ADJ_N3], e = u[4*ADJ_N3];
         floored = a.ph.min_pres > eint_con<P>( d, 1.f/d, m1, m2, m3, e )*a.ph.gm1;
      }
      const double v1 = (double)w[AF_N2], v2 = (double)w[2*AF_N2], v3 = (double)w[3*AF_N2], ir = rcp_dd( (double)w[0] );
      const double pb = floored ? 0.0 : wb[4]*(double)a.ph.gm1;
      out[0] += wb[0] - ( wb[1]*v1 + wb[2]*v2 + wb[3]*v3 )*ir + 0.5*pb*( v1*v1 + v2*v2 + v3*v3 );
      out[1] += wb[1]*ir - pb*v1;
      out[2] += wb[2]*ir - pb*v2;
      out[3] += wb[3]*ir - pb*v3;
      out[4] += pb;
   }
   if ( g != nullptr )
   {
#     pragma unroll
      for (int v=0; v<ADJ_NC; v++) out[v] += g[v*PS2*PS2];
   }
#  pragma unroll
   for (int v=0; v<ADJ_NC; v++) gi[v*ADJ_N3] = out[v];
}

// the cell adjoint of one direction: bl, br the adjoints of the two faces; the part of the cell itself is added to
// cen, put( v, lo, hi ) takes those for the cells below and above it
template <int D, typename F>
GB_DEV void adj_dir( const AdjArgs<float> &a, const float *wm, const float *wc, const float *wp, const double (&bl)[ADJ_NC],
                     const double (&br)[ADJ_NC], const double (&accbar)[ADJ_NC], double (&cen)[ADJ_NC], const F &put )
{
   float fl[ADJ_NC], fr[ADJ_NC];
   int code[ADJ_NC];
   adj_faces<D>( wm, wc, wp, a.coeff, fl, fr, code );
   // F_{2d} enters the Hancock sum with -, F_{2d+1} with +
   double wbl[ADJ_NC], wbr[ADJ_NC];
   adj_face_prim<D>( a.ph, fl, bl, -1.0, accbar, wbl );
   adj_face_prim<D>( a.ph, fr, br,  1.0, accbar, wbr );
   // face values C -+ S/2: the slope takes half the difference of the two adjoints
#  pragma unroll
   for (int v=0; v<ADJ_NC; v++)
   {
      float sl, sc, sr;
      gminmod_partials( code[v], a.coeff, sl, sc, sr );
      const double sb = 0.5*( wbr[v] - wbl[v] );
      cen[v] += ( wbl[v] + wbr[v] ) + (double)sc*sb;
      put( v, (double)sl*sb, (double)sr*sb );
   }
}

// nan_pg[npg]: set (RESCUE false) to whether a flux of the patch group came out NaN; those patch groups are
// done again by the instantiation with RESCUE true, whose call for such faces costs the other one
// its registers (1.1 KB of spills)
template <int P, bool RESCUE>
__global__ void __launch_bounds__( AF_THREADS, 1 ) adj_fused_kernel( const __grid_constant__ AdjArgs<float> a, int *nan_pg, int *status )
{
   typedef AdjFusedSmem S;
   constexpr int N = ADJ_N, NF = ADJ_F, NC = ADJ_NC, OUT2 = PS2*PS2, O3 = PS2*PS2*PS2;
   extern __shared__ __align__(128) unsigned char smem[];
   uint64_t *bar = (uint64_t*)smem;
   int *s_abort  = (int*)( smem + 96 ), *s_nan = (int*)( smem + 100 );
   float  *s_ring = (float*)( smem + S::o_ring ), *s_fc = (float*)( smem + S::o_fc );
   double *s_q = (double*)( smem + S::o_q ), *s_c = (double*)( smem + S::o_c ), *s_g = (double*)( smem + S::o_g );
   double *s_z = (double*)( smem + S::o_z );
   const int tid = threadIdx.x, nth = AF_THREADS;
   const Phys<float> ph = a.ph;
   const float dt_dh2 = 0.5f*a.dt/a.dh;
   const double dtdh = (double)a.dt/(double)a.dh, k2 = 0.5*(double)a.dt/(double)a.dh;
   if ( tid == 0 )
   {
      for (int q=0; q<AF_SLOTS + AF_GSLOTS; q++) mbar_init( &bar[q], 1 );
      mbar_init_fence();
      *s_abort = 0;
      *s_nan = 0;
   }
   for (int e = tid; e < NC*AF_FACES; e += nth) s_z[e] = 0.0;
   __syncthreads();

   int i, j;
   const bool col = ( tid < AF_CELLS ), inner = ( tid < OUT2 );
   if ( inner ) { i = 1 + tid % PS2;  j = 1 + tid / PS2; }
   else
   {
      const int h = tid - OUT2;
      if      ( h < NF )          { i = h;      j = 0;      }
      else if ( h < 2*NF )        { i = h - NF; j = NF - 1; }
      else if ( h < 2*NF + PS2 )  { i = 0;      j = 1 + h - 2*NF; }
      else                        { i = NF - 1; j = ( 1 + h - 2*NF - PS2 < NF ) ? 1 + h - 2*NF - PS2 : NF - 1; }
   }
   const bool in_i = ( i >= 1 && i <= PS2 ), in_j = ( j >= 1 && j <= PS2 );
   const int f = j*NF + i, cell = ( j + 1 )*N + i + 1;

   // the adjoints of this cell's lower and upper x and y face states (those of absent faces are zero)
   const double *qxl = ( in_j && i >= 1 )   ? s_q + 1*NC*AF_FACES + ( j - 1 )*NFLX + i - 1 : s_z;
   const double *qxu = ( in_j && i <= PS2 ) ? s_q + ( j - 1 )*NFLX + i : s_z;
   const double *qyl = ( in_i && j >= 1 )   ? s_q + 3*NC*AF_FACES + ( j - 1 )*PS2 + i - 1 : s_z;
   const double *qyu = ( in_i && j <= PS2 ) ? s_q + 2*NC*AF_FACES + j*PS2 + i - 1 : s_z;

   // every patch group uses each ring slot four times, so plane c's wait has the parity of c/5 (of c/4)
   static_assert( N % AF_SLOTS == 0 && ( N/AF_SLOTS ) % 2 == 0 && PS2 % AF_GSLOTS == 0 && ( PS2/AF_GSLOTS ) % 2 == 0, "ring parity" );
   auto parity = [&]( int c ) { return (uint32_t)( c/AF_SLOTS ) & 1u; };

   for (int pgi = blockIdx.x; pgi < a.npg; pgi += gridDim.x)
   {
      if ( RESCUE && nan_pg[pgi] == 0 ) continue;
      const size_t pg = pgi;
      const float *g_in = a.in + pg*NC*ADJ_N3;
      const double *g_out = a.gout + pg*NC*O3;
      auto issue = [&]( int c ) {
         if ( c >= N ) return;
         const int q = c % AF_SLOTS;
         fence_proxy_async();
         mbar_expect_tx( &bar[q], AF_PLANE*4 );
         for (int v=0; v<NC; v++) bulk_g2s( s_ring + q*AF_PLANE + v*AF_N2, g_in + (size_t)v*ADJ_N3 + (size_t)c*AF_N2, AF_N2*4, &bar[q] );
      };
      // planes of d loss / d U_out: plane o is used from face-state plane o+1 on, last by the input plane o+2
      auto issue_g = [&]( int o ) {
         if ( o >= PS2 ) return;
         const int q = o % AF_GSLOTS;
         fence_proxy_async();
         mbar_expect_tx( &bar[AF_SLOTS + q], NC*OUT2*8 );
         for (int v=0; v<NC; v++) bulk_g2s( s_g + ( q*NC + v )*OUT2, g_out + (size_t)v*O3 + (size_t)o*OUT2, OUT2*8, &bar[AF_SLOTS + q] );
      };
      auto wait_g = [&]( int o ) {
         if ( o >= PS2 ) return;
         if ( !mbar_wait_bounded( &bar[AF_SLOTS + o % AF_GSLOTS], (uint32_t)( o/AF_GSLOTS ) & 1u ) )
         {
            atomicOr( status, GB_ST_TMA_TIMEOUT );
            *s_abort = 1;
         }
      };
      auto gplane = [&]( int o ) { return s_g + ( o % AF_GSLOTS )*NC*OUT2; };
      auto convert = [&]( int c, int vt ) {
         if ( c >= N ) return;
         if ( !mbar_wait_bounded( &bar[c % AF_SLOTS], parity( c ) ) )
         {
            atomicOr( status, GB_ST_TMA_TIMEOUT );
            *s_abort = 1;
         }
         float2 *w2 = (float2*)( s_ring + ( c % AF_SLOTS )*AF_PLANE );
         for (int e = vt; e < AF_N2/2; e += nth)
         {
            float2 u[NC], w[NC];
#           pragma unroll
            for (int v=0; v<NC; v++) u[v] = w2[v*( AF_N2/2 ) + e];
            con2pri_pair<P,NC>( ph, u, w );
#           pragma unroll
            for (int v=0; v<NC; v++) w2[v*( AF_N2/2 ) + e] = w[v];
         }
      };
      auto ring = [&]( int c ) { return s_ring + ( c % AF_SLOTS )*AF_PLANE + cell; };

      if ( tid == 0 )
      {
         for (int c=0; c<AF_SLOTS; c++) issue( c );
         for (int o=0; o<AF_GSLOTS; o++) issue_g( o );
      }
      for (int c=0; c<3; c++) convert( c, tid );
      __syncthreads();
      if ( *s_abort ) { if ( tid == 0 ) for (int c=0; c<AF_SLOTS + AF_GSLOTS; c++) mbar_wait_bounded( &bar[c], 0 );  __syncthreads();  return; }

      // carried by the column: the upper z face state and the reset flag of plane k-1, the adjoint of that plane's
      // lower z face, and the sums of input planes k-1 (acc0) and k (acc1); ext: gin of plane k-1
      // holds a reset part
      float  zup[NC] = { 0.f, 0.f, 0.f, 0.f, 0.f };
      double rbz[NC], acc0[NC], acc1[NC];
#     pragma unroll
      for (int v=0; v<NC; v++) rbz[v] = acc0[v] = acc1[v] = 0.0;
      bool rst = false, ext = false;

      for (int k=0; k<=N; k++)
      {
         if ( col )
         {
            // face states of plane k
            float zl[NC], zu[NC];
            bool rst_k = false;
#           pragma unroll
            for (int v=0; v<NC; v++) zl[v] = zu[v] = 0.f;
            if ( k < NF )
            {
               const float *pc = ring( k + 1 ), *pm = ring( k ), *pp = ring( k + 2 );
               float cc[NC], nl[NC], nr[NC], fpres[6], acc[NC];
               float2 fc[3][NC];
#              pragma unroll
               for (int v=0; v<NC; v++) { cc[v] = pc[v*AF_N2];  nl[v] = pc[v*AF_N2 - 1];  nr[v] = pc[v*AF_N2 + 1]; }
               recon_dir_pair<0,P,NC,false>( ph, cc, nl, nr, LIM_GMINMOD, a.coeff, false, fc, fpres, acc );
#              pragma unroll
               for (int v=0; v<NC; v++) { nl[v] = pc[v*AF_N2 - N];  nr[v] = pc[v*AF_N2 + N]; }
               recon_dir_pair<1,P,NC,false>( ph, cc, nl, nr, LIM_GMINMOD, a.coeff, false, fc, fpres, acc );
#              pragma unroll
               for (int v=0; v<NC; v++) { nl[v] = pm[v*AF_N2];  nr[v] = pp[v*AF_N2]; }
               recon_dir_pair<2,P,NC,false>( ph, cc, nl, nr, LIM_GMINMOD, a.coeff, false, fc, fpres, acc );
               hancock_finish_pair<P,NC>( ph, dt_dh2, fc, fpres, acc, g_in + (size_t)( k + 1 )*AF_N2 + cell, (size_t)ADJ_N3, rst_k );
               float *sx = s_fc + f, *sy = sx + 2*NC*AF_CELLS;
#              pragma unroll
               for (int v=0; v<NC; v++)
               {
                  sx[v*AF_CELLS] = fc[0][v].x;  sx[( NC + v )*AF_CELLS] = fc[0][v].y;
                  sy[v*AF_CELLS] = fc[1][v].x;  sy[( NC + v )*AF_CELLS] = fc[1][v].y;
                  zl[v] = fc[2][v].x;  zu[v] = fc[2][v].y;
               }
            }
            // the z Riemann problem between planes k-1 and k
            double zb[NC], rb[NC];                   // adjoints of the face states below and above it
#           pragma unroll
            for (int v=0; v<NC; v++) zb[v] = rb[v] = 0.0;
            if ( inner && k >= 1 && k < NF )
            {
               const int ko = k - 1;
               double fbar[NC];
#              pragma unroll
               for (int v=0; v<NC; v++)
               {
                  fbar[v] = dtdh*( ( ko < PS2 ? gplane( ko )[v*OUT2 + tid] : 0.0 ) - ( ko >= 1 ? gplane( ko - 1 )[v*OUT2 + tid] : 0.0 ) );
               }
               adj_face_hllc<2,P,RESCUE>( ph, zup, zl, fbar, zb, rb, s_nan );
            }
            // the cell adjoint of plane k-1: its own part is added to acc1, the ones along z to acc0 and zhi
            double zhi[NC];
#           pragma unroll
            for (int v=0; v<NC; v++) zhi[v] = 0.0;
            bool ext_k = false;
            if ( k >= 1 && k <= NF )
            {
               const bool plane = ( k >= 2 && k <= NF - 1 );         // x and y faces
               const double *x0 = plane ? qxl : s_z, *x1 = plane ? qxu : s_z, *y0 = plane ? qyl : s_z, *y1 = plane ? qyu : s_z;
               double s[NC];
               bool any = false;
#              pragma unroll
               for (int v=0; v<NC; v++)
               {
                  const double q0 = x0[v*AF_FACES], q1 = x1[v*AF_FACES], q2 = y0[v*AF_FACES], q3 = y1[v*AF_FACES];
                  s[v] = ( ( ( ( q0 + q1 ) + q2 ) + q3 ) + rbz[v] ) + zb[v];
                  any |= ( q0 != 0.0 || q1 != 0.0 || q2 != 0.0 || q3 != 0.0 || rbz[v] != 0.0 || zb[v] != 0.0 );
               }
               double *cx = s_c + f;
               if ( any && rst )
               {
                  // MHM_CHECK_PREDICT reset: every face state was the cell's input value
                  double *gi = a.gin + pg*NC*ADJ_N3 + (size_t)k*AF_N2 + cell;
#                 pragma unroll
                  for (int v=0; v<NC; v++) gi[v*ADJ_N3] = s[v];
                  ext_k = true;
               }
               if ( any && !rst )
               {
                  // Hancock: q_f = u_f - k2 acc, so ubar_f = qbar_f and accbar = -k2 sum_f qbar_f
                  double accbar[NC], bl[NC], br[NC];
                  const float *pc = ring( k ), *pm = ring( k - 1 ), *pp = ring( k + 1 );
                  float wc[NC], wm[NC], wp[NC];
#                 pragma unroll
                  for (int v=0; v<NC; v++) { accbar[v] = -k2*s[v];  wc[v] = pc[v*AF_N2];  wm[v] = pm[v*AF_N2];  wp[v] = pp[v*AF_N2]; }
                  adj_dir<2>( a, wm, wc, wp, rbz, zb, accbar, acc1, [&]( int v, double lo, double hi ) { acc0[v] += lo;  zhi[v] = hi; } );
#                 pragma unroll
                  for (int v=0; v<NC; v++)
                  {
                     wm[v] = pc[v*AF_N2 - 1];  wp[v] = pc[v*AF_N2 + 1];
                     bl[v] = x0[v*AF_FACES];  br[v] = x1[v*AF_FACES];
                  }
                  adj_dir<0>( a, wm, wc, wp, bl, br, accbar, acc1,
                              [&]( int v, double lo, double hi ) { cx[v*AF_CELLS] = lo;  cx[( NC + v )*AF_CELLS] = hi; } );
#                 pragma unroll
                  for (int v=0; v<NC; v++)
                  {
                     wm[v] = pc[v*AF_N2 - N];  wp[v] = pc[v*AF_N2 + N];
                     bl[v] = y0[v*AF_FACES];  br[v] = y1[v*AF_FACES];
                  }
                  adj_dir<1>( a, wm, wc, wp, bl, br, accbar, acc1,
                              [&]( int v, double lo, double hi ) { cx[( 2*NC + v )*AF_CELLS] = lo;  cx[( 3*NC + v )*AF_CELLS] = hi; } );
               }
               else
               {
#                 pragma unroll
                  for (int q=0; q<4*NC; q++) cx[q*AF_CELLS] = 0.0;
               }
            }
            // input plane k-1 is complete
            if ( k >= 1 )
            {
               const int o = k - 3;
               adj_cell_out<P>( a, pg, ( k - 1 )*AF_N2 + cell, acc0, ring( k - 1 ), ext, ( inner && o >= 0 && o < PS2 ) ? gplane( o ) + tid : nullptr );
            }
#           pragma unroll
            for (int v=0; v<NC; v++)
            {
               acc0[v] = acc1[v];
               acc1[v] = zhi[v];
               rbz[v]  = rb[v];
               zup[v]  = zu[v];
            }
            rst = rst_k;
            ext = ext_k;
         }
         __syncthreads();
         if ( tid == 0 && k >= 1 )
         {
            issue( k + 4 );                            // the slot of input plane k-1
            if ( k >= 3 ) issue_g( k + 1 );            // and of output plane k-3
         }
         if ( k == N ) break;

         // the x and y Riemann problems of plane k
         int nitem = 0;
         if ( k >= 1 && k <= PS2 )
         {
            nitem = 2*AF_FACES;
            for (int e = tid; e < nitem; e += nth)
            {
               const bool yd = ( e >= AF_FACES );
               const int e1 = yd ? e - AF_FACES : e;
               const int fi = yd ? 1 + e1 % PS2 : e1 % NFLX, fj = yd ? e1 / PS2 : 1 + e1 / NFLX;
               const float *sd = s_fc + ( yd ? 2*NC*AF_CELLS : 0 ) + fj*NF + fi;
               const int step = yd ? NF : 1, gs = yd ? PS2 : 1, nrm = yd ? fj : fi;
               // the rotated frame: density, normal, two transverse momenta, energy
               float L[NC], Rr[NC];
               double fbar[NC], lb[NC], rb[NC];
               const double *g = gplane( k - 1 ) + ( fj - 1 )*PS2 + fi - 1;             // the output cell below the face
               // the rotated momenta 1..3 are the components y, z, x of a y face
#              pragma unroll
               for (int q=0; q<NC; q++)
               {
                  const int v = ( yd && q >= 1 && q <= 3 ) ? ( q == 3 ? 1 : q + 1 ) : q;
                  L[q]  = sd[( NC + v )*AF_CELLS];
                  Rr[q] = sd[v*AF_CELLS + step];
                  fbar[q] = dtdh*( ( nrm < PS2 ? g[v*OUT2 + gs] : 0.0 ) - ( nrm >= 1 ? g[v*OUT2] : 0.0 ) );
               }
               adj_face_hllc<0,P,RESCUE>( ph, L, Rr, fbar, lb, rb, s_nan );
               double *q0 = s_q + ( yd ? 2*NC*AF_FACES : 0 ) + e1;
#              pragma unroll
               for (int q=0; q<NC; q++)
               {
                  const int v = ( yd && q >= 1 && q <= 3 ) ? ( q == 3 ? 1 : q + 1 ) : q;
                  q0[v*AF_FACES] = lb[q];  q0[( NC + v )*AF_FACES] = rb[q];
               }
            }
         }
         // the neighbours' parts of input plane k (from face-state plane k-1)
         const bool parts = ( k >= 1 && k <= NF );
         if ( parts && col )
         {
#           pragma unroll
            for (int v=0; v<NC; v++)
            {
               const double *c = s_c + v*AF_CELLS + f;
               double t = acc0[v];
               if ( i < NF - 1 ) t += c[1];
               if ( i > 0 )      t += c[NC*AF_CELLS - 1];
               if ( j < NF - 1 ) t += c[2*NC*AF_CELLS + NF];
               if ( j > 0 )      t += c[3*NC*AF_CELLS - NF];
               acc0[v] = t;
            }
         }
         // the input cells of plane k around the columns
         for (int b = ( tid + nth - nitem % nth ) % nth; b < AF_BORDER; b += nth)
         {
            int bi, bj;
            if      ( b < N )         { bi = b;         bj = 0;     }
            else if ( b < 2*N )       { bi = b - N;     bj = N - 1; }
            else if ( b < 3*N - 2 )   { bi = 0;         bj = 1 + b - 2*N; }
            else                      { bi = N - 1;     bj = 1 + b - ( 3*N - 2 ); }
            double wb[NC] = { 0.0, 0.0, 0.0, 0.0, 0.0 };
            const bool mid_i = ( bi >= 1 && bi <= NF ), mid_j = ( bj >= 1 && bj <= NF );
            if ( parts && ( mid_i || mid_j ) )
            {
               const int dir = mid_j ? ( bi == 0 ? 0 : 1 ) : ( bj == 0 ? 2 : 3 );
               const int fb = mid_j ? ( bj - 1 )*NF + ( bi == 0 ? 0 : NF - 1 ) : ( bj == 0 ? 0 : NF - 1 )*NF + bi - 1;
#              pragma unroll
               for (int v=0; v<NC; v++) wb[v] = s_c[( dir*NC + v )*AF_CELLS + fb];
            }
            adj_cell_out<P>( a, pg, k*AF_N2 + bj*N + bi, wb, s_ring + ( k % AF_SLOTS )*AF_PLANE + bj*N + bi, false, nullptr );
         }
         convert( k + 3, ( tid + 2*nth - ( nitem + AF_BORDER ) % nth ) % nth );
         wait_g( k );
         __syncthreads();
         if ( *s_abort )
         {
            // wait once more (bounded) for the copies that may be in flight, then give up
            if ( tid == 0 )
            {
               if ( k + 4 < N ) mbar_wait_bounded( &bar[( k + 4 ) % AF_SLOTS], parity( k + 4 ) );
               for (int o = k + 1; o <= k + 3 && o < PS2; o++)
                  if ( o <= ( k >= 3 ? k + 1 : AF_GSLOTS - 1 ) ) mbar_wait_bounded( &bar[AF_SLOTS + o % AF_GSLOTS], (uint32_t)( o/AF_GSLOTS ) & 1u );
            }
            __syncthreads();
            return;
         }
      }
      if ( !RESCUE && tid == 0 ) { nan_pg[pgi] = *s_nan;  *s_nan = 0; }
      __syncthreads();
   }
}

} // namespace gb
