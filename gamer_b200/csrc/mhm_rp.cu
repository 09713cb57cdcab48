// MHM_RP half step (hydro): Hydro_RiemannPredict_Flux + Hydro_RiemannPredict
// (src/Model_Hydro/CPU_Hydro/CPU_FluidSolver_MHM.cpp:593-950).
//
// The reference evaluates first-order Riemann fluxes between neighbouring input cells over the
// whole 22^3 window, stores them in global scratch (g_Flux_Half), then advances the inner 20^3
// cells by dt/2 with them and stores the primitive half-step state (g_PriVar_Half) for the PLM
// reconstruction of the full step (22^3 -> 20^3 with PLM, 24^3 -> 22^3 with PPM).  Here one CTA
// sweeps a patch group plane by plane along z:
//   * the conserved input planes kc-1..kc+1 stay in a three-plane ring in shared memory;
//   * for half-step plane k (input plane kc = k+1) it solves the z problems between kc and kc+1
//     (20x20), the x problems of plane kc (21 faces x 20 rows) and the y problems (20 columns x 21
//     faces) -- 1240 per plane -- into shared-memory flux planes; the z fluxes below, between kc-1
//     and kc, are the previous plane's;
//   * each half-step cell is then U_in - dt/(2dh) * ((dFx + dFy) + dFz) (the reference's summation
//     order), floored (MinDens, MinEint, PassiveFloor), converted to primitive variables (with the
//     Jeans pressure floor and FracPassive) and written to the half-step state [npg][NC][20^3], which
//     the MHM kernel's SCH_MHM_RP instantiation reconstructs from.
// Every Riemann problem is solved once; the global traffic is the input read once and the half-step
// state written once.  The mixed policy accumulates the flux differences in double.
#include <cstring>
#include <type_traits>
#include <cuda_runtime.h>
#include "../../include/gamer_b200_fluid.h"
#include "hydro_physics.cuh"
#include "tma.cuh"

namespace gb {

template <typename R>
struct RpArgs {
   const R *in;       // [npg][NC][N^3] conserved (N = 22 with PLM, 24 with PPM)
   R       *half;     // [npg][NC][(N-2)^3] primitive half-step state
   int      npg;
   R        dt_dh2;   // dt/(2 dh)
   int     *status;   // one status word, GB_ST_* bits OR-ed in
   int      nitem, nwhole, nslab;   // work items: the patch groups below nwhole whole, the others in nslab slabs
   Phys<R>  ph;
};

// input width NXI (FLU_NXT: 22 with PLM, 24 with PPM), flux faces NXI - 1, half-state width NXI - 2
constexpr int RPH_BLOCK = 256;

__host__ __device__ inline size_t rp_half_smem( int rsz, int nc, int nxi )
{
   const int nf = nxi - 1, nv = nxi - 2;
   return (size_t)rsz*nc*( 3*nxi*nxi + 2*nv*nv + 2*nv*nf );
}

template <typename R, int P, int RS, int NC, int NXI>
__global__ void __launch_bounds__( RPH_BLOCK ) mhm_rp_half_kernel( const __grid_constant__ RpArgs<R> a )
{
   typedef typename std::conditional<P == P_MIXED, double, R>::type A;   // accumulation type
   constexpr int N = NXI, NF = NXI - 1, NV = NXI - 2, N2 = N*N, NV2 = NV*NV, NV3 = NV*NV*NV;
   constexpr int NZ = NV2, NXF = NV*NF;          // z problems, x (and y) problems per plane
   extern __shared__ __align__(16) unsigned char smem[];
   R *s_in = (R*)smem;                   // [3][NC][N*N]  conserved planes, slot = plane % 3
   R *s_fz = s_in + 3*NC*N2;             // [2][NC][NV][NV] z fluxes, slot = (upper input plane) & 1
   R *s_fx = s_fz + 2*NC*NV2;            // [NC][NV rows j-1][NF faces i]
   R *s_fy = s_fx + NC*NXF;              // [NC][NF faces j][NV columns i-1]
   const int tid = threadIdx.x, nth = blockDim.x;
   const Phys<R> ph = a.ph;

   for (int pg = blockIdx.x; pg < a.npg; pg += gridDim.x)
   {
      const R *g = a.in + (size_t)pg*NC*N*N2;
      R *h = a.half + (size_t)pg*NC*NV3;

      auto load = [&]( int c ) {
         R *dst = s_in + ( c % 3 )*NC*N2;
         for (int e = tid; e < NC*N2; e += nth)
         {
            const int v = e / N2, r = e % N2;
            dst[e] = g[(size_t)v*N*N2 + (size_t)c*N2 + r];
         }
      };
      // z problems between input planes c and c+1 at columns (i, j) = 1..NV, into slot (c+1) & 1
      auto zflux = [&]( int c, int e ) {
         const R *lo = s_in + ( c % 3 )*NC*N2, *hi = s_in + ( ( c + 1 ) % 3 )*NC*N2;
         const int i = 1 + e % NV, j = 1 + e / NV, q = j*N + i;
         R L[NC], Rr[NC], F[NC];
#        pragma unroll
         for (int v=0; v<NC; v++) { L[v] = lo[v*N2 + q];  Rr[v] = hi[v*N2 + q]; }
         riemann<RS,2,P,NC>( ph, L, Rr, F );
         R *dst = s_fz + ( ( c + 1 ) & 1 )*NC*NV2 + e;
#        pragma unroll
         for (int v=0; v<NC; v++) dst[v*NV2] = F[v];
      };

      __syncthreads();                    // the previous patch group's last reads are done
      load( 0 );
      load( 1 );
      __syncthreads();
      for (int e = tid; e < NZ; e += nth) zflux( 0, e );

      for (int k = 0; k < NV; k++)
      {
         const int kc = k + 1;            // input plane of half-step plane k
         load( kc + 1 );                  // its slot held plane kc-2, no longer read
         __syncthreads();
         // the z problems above plane kc and the x / y problems of plane kc
         const R *pc = s_in + ( kc % 3 )*NC*N2;
         for (int e = tid; e < NZ + 2*NXF; e += nth)
         {
            if ( e < NZ ) { zflux( kc, e );  continue; }
            R L[NC], Rr[NC], F[NC];
            if ( e < NZ + NXF )
            {
               const int f = e - NZ, i = f % NF, j = 1 + f / NF, q = j*N + i;   // face between i and i+1
#              pragma unroll
               for (int v=0; v<NC; v++) { L[v] = pc[v*N2 + q];  Rr[v] = pc[v*N2 + q + 1]; }
               riemann<RS,0,P,NC>( ph, L, Rr, F );
#              pragma unroll
               for (int v=0; v<NC; v++) s_fx[v*NXF + f] = F[v];
            }
            else
            {
               const int f = e - NZ - NXF, i = 1 + f % NV, j = f / NV, q = j*N + i;   // face between j and j+1
#              pragma unroll
               for (int v=0; v<NC; v++) { L[v] = pc[v*N2 + q];  Rr[v] = pc[v*N2 + q + N]; }
               riemann<RS,1,P,NC>( ph, L, Rr, F );
#              pragma unroll
               for (int v=0; v<NC; v++) s_fy[v*NXF + f] = F[v];
            }
         }
         __syncthreads();
         // half-step cells of plane k
         const R *fzl = s_fz + ( kc & 1 )*NC*NV2, *fzu = s_fz + ( ( kc + 1 ) & 1 )*NC*NV2;
         for (int e = tid; e < NV2; e += nth)
         {
            const int i = e % NV, j = e / NV, q = ( j + 1 )*N + ( i + 1 );
            R u[NC], w[NC];
#           pragma unroll
            for (int v=0; v<NC; v++)
            {
               const A dfx = (A)s_fx[v*NXF + j*NF + i + 1] - (A)s_fx[v*NXF + j*NF + i];
               const A dfy = (A)s_fy[v*NXF + ( j + 1 )*NV + i] - (A)s_fy[v*NXF + j*NV + i];
               const A dfz = (A)fzu[v*NV2 + e] - (A)fzl[v*NV2 + e];
               u[v] = (R)( (A)pc[v*N2 + q] - (A)a.dt_dh2*( ( dfx + dfy ) + dfz ) );
            }
            u[0] = gmax( u[0], ph.min_dens );
            u[4] = floor_eint_in_engy<P>( ph, u[0], u[1], u[2], u[3], u[4] );
#           pragma unroll
            for (int v=5; v<NC; v++) if ( ph.pfloor & ( 1u << v ) ) u[v] = gmax( u[v], Lim<R>::tiny() );
            con2pri_cc<P,NC>( ph, u, w );
#           pragma unroll
            for (int v=0; v<NC; v++) h[(size_t)v*NV3 + (size_t)k*NV2 + e] = w[v];
         }
         // the next iteration's load writes the slot of plane kc-1 (not read here) and its
         // barrier orders these reads of s_fx / s_fy / s_fz before the next writes
      }
   }
}

// ---- the float policies' half step with HLLC and five variables ------------------------------------
// Every state of a first-order problem is an input cell, met by six problems, so its reciprocal
// density, pressure and sound speed are formed once per cell and kept beside it in the plane ring.
// One barrier per plane: in step c the thread of column (i, j) solves the z problem between planes c
// and c+1, with the flux below plane c carried in registers, and advances its half-step cell of plane
// c with the x and y fluxes of the step before; an x face and a y face of plane c+1 are the lanes of
// one packed HLLC, into the other of two flux buffers; and plane c+2 is prepared while plane c+3
// arrives by 1-D bulk copies.  The sums are those of mhm_rp_half_kernel.
// 22-wide planes: 448 threads (20 x 20 columns, 420 face pairs), two CTAs per SM (72 registers, 98 KB);
// 24-wide: 512 threads (484, 506), one CTA (114 KB).  729 patch groups, mixed, with the full step:
// 545 -> 389 us; 8 patch groups: 151 -> 24 us.  The patch groups of the last, partly filled wave go in slabs of planes, as in mhm_plan.
template <int NXI> struct RpxSmem {
   static constexpr int NV = NXI - 2, NF = NXI - 1, N2 = NXI*NXI, NXF = NV*NF;
   static constexpr int THREADS = ( NXI == 22 ) ? 448 : 512, CTAS = ( NXI == 22 ) ? 2 : 1;
   static constexpr int SLOT = 8*N2;                 // 5 conserved variables, 1/rho, P, c_s
   static constexpr int o_ring = 64, o_fl = o_ring + 4*SLOT*4;
   static constexpr int bytes = o_fl + 2*2*5*NXF*4;  // [2 buffers][x, y][5][faces]
};

template <int P, int NXI>
__global__ void __launch_bounds__( RpxSmem<NXI>::THREADS, RpxSmem<NXI>::CTAS ) rp_half_hllc_kernel( const __grid_constant__ RpArgs<float> a )
{
   typedef RpxSmem<NXI> S;
   typedef typename std::conditional<P == P_MIXED, double, float>::type A;   // accumulation type
   constexpr int N = NXI, N2 = S::N2, NV = S::NV, NF = S::NF, NXF = S::NXF, NV2 = NV*NV, NV3 = NV2*NV, SLOT = S::SLOT;
   constexpr int NX3 = NXI*NXI*NXI;
   static_assert( NXF <= S::THREADS && NV2 <= S::THREADS, "one column and one face pair per thread" );
   extern __shared__ __align__(128) unsigned char smem[];
   uint64_t *bar = (uint64_t*)smem;
   int *s_abort  = (int*)( smem + 48 );
   float *s_ring = (float*)( smem + S::o_ring ), *s_fl = (float*)( smem + S::o_fl );
   const int tid = threadIdx.x, nth = S::THREADS;
   const Phys<float> ph = a.ph;
   const A k2 = (A)a.dt_dh2;
   if ( tid == 0 )
   {
      for (int q=0; q<4; q++) mbar_init( &bar[q], 1 );
      mbar_init_fence();
      *s_abort = 0;
   }
   __syncthreads();
   uint32_t phase = 0;                               // bit q: parity of slot q's next use
   for (int item = blockIdx.x; item < a.nitem; item += gridDim.x)
   {
      // half-step planes [o0, o0 + np) of the patch group: input planes o0 .. o0 + np + 1, numbered from 0
      const bool whole = ( item < a.nwhole );
      const int part = item - a.nwhole, pg = whole ? item : a.nwhole + part/a.nslab;
      const int np = whole ? NV : NV/a.nslab, o0 = whole ? 0 : ( part % a.nslab )*np, nz = np + 2;
      const float *g = a.in + (size_t)pg*5*NX3 + (size_t)o0*N2;
      float *h = a.half + (size_t)pg*5*NV3 + (size_t)o0*NV2;
      auto issue = [&]( int c ) {
         if ( c >= nz ) return;
         const int q = c & 3;
         fence_proxy_async();
         mbar_expect_tx( &bar[q], 5*N2*4 );
         for (int v=0; v<5; v++) bulk_g2s( s_ring + q*SLOT + v*N2, g + (size_t)v*NX3 + (size_t)c*N2, N2*4, &bar[q] );
      };
      // wait for plane c and form 1/rho, P and c_s of its cells; the caller is number vt of the threads
      auto derive = [&]( int c, int vt ) {
         if ( c >= nz ) return;
         if ( !mbar_wait_bounded( &bar[c & 3], ( ( phase >> ( c & 3 ) ) + (uint32_t)( c >> 2 ) ) & 1u ) )
         {
            atomicOr( a.status, GB_ST_TMA_TIMEOUT );
            *s_abort = 1;
         }
         float2 *w = (float2*)( s_ring + ( c & 3 )*SLOT );
         constexpr int H = N2/2;
         for (int e = vt; e < H; e += nth)
         {
            const float2 d = w[e], ir = make_float2( 1.f/d.x, 1.f/d.y );
            const float2 p = pres_con_pair<P>( ph, d, ir, w[H + e], w[2*H + e], w[3*H + e], w[4*H + e] );
            const float2 c2 = p_mul( p_mul( p_bc( ph.gamma ), p ), ir );
            w[5*H + e] = ir;  w[6*H + e] = p;  w[7*H + e] = make_float2( sqrtf( c2.x ), sqrtf( c2.y ) );
         }
      };
      // x face e (between columns i and i+1) and y face e of plane c, into flux buffer c & 1
      auto faces = [&]( int c ) {
         constexpr int ry[5] = { 0, 2, 3, 1, 4 };
         const float *w = s_ring + ( c & 3 )*SLOT;
         float *fx = s_fl + ( c & 1 )*10*NXF, *fy = fx + 5*NXF;
         if ( const int e = tid; e < NXF )
         {
            const int qx = ( 1 + e / NF )*N + e % NF, qy = ( e / NV )*N + 1 + e % NV;
            float2 L[5], Rr[5], F[5];
#           pragma unroll
            for (int v=0; v<5; v++)
            {
               L[v]  = make_float2( w[v*N2 + qx],     w[ry[v]*N2 + qy] );
               Rr[v] = make_float2( w[v*N2 + qx + 1], w[ry[v]*N2 + qy + N] );
            }
            bool nan_x, nan_y;
            hllc_x2_core( ph, L, Rr, make_float2( w[5*N2 + qx], w[5*N2 + qy] ), make_float2( w[5*N2 + qx + 1], w[5*N2 + qy + N] ),
                          make_float2( w[6*N2 + qx], w[6*N2 + qy] ), make_float2( w[6*N2 + qx + 1], w[6*N2 + qy + N] ),
                          make_float2( w[7*N2 + qx], w[7*N2 + qy] ), make_float2( w[7*N2 + qx + 1], w[7*N2 + qy + N] ),
                          F, nan_x, nan_y );
            float Fx[5], Fy[5];
#           pragma unroll
            for (int v=0; v<5; v++) { Fx[v] = F[v].x;  Fy[ry[v]] = F[v].y; }
            if ( nan_x || nan_y )
            {
               // HLLE rescue of a NaN flux (CPU_Shared_ComputeFlux.cpp:313-362), per face
               float l[5], r[5];
               if ( nan_x )
               {
#                 pragma unroll
                  for (int v=0; v<5; v++) { l[v] = L[v].x;  r[v] = Rr[v].x; }
                  riemann_hlle_outlined<0,P,5>( ph, l, r, Fx );
               }
               if ( nan_y )
               {
#                 pragma unroll
                  for (int v=0; v<5; v++) { l[ry[v]] = L[v].y;  r[ry[v]] = Rr[v].y; }
                  riemann_hlle_outlined<1,P,5>( ph, l, r, Fy );
               }
            }
#           pragma unroll
            for (int v=0; v<5; v++) { fx[v*NXF + e] = Fx[v];  fy[v*NXF + e] = Fy[v]; }
         }
      };

      if ( tid == 0 ) for (int c=0; c<4; c++) issue( c );
      derive( 0, tid );
      derive( 1, tid );
      __syncthreads();
      if ( *s_abort ) { if ( tid == 0 ) for (int c=2; c<4 && c<nz; c++) mbar_wait_bounded( &bar[c], ( phase >> c ) & 1u );  __syncthreads();  return; }
      float fzl[5] = { 0.f, 0.f, 0.f, 0.f, 0.f };   // z flux below the column's cell
      for (int c=0; c<=np; c++)
      {
         const float *w0 = s_ring + ( c & 3 )*SLOT, *w1 = s_ring + ( ( c + 1 ) & 3 )*SLOT;
         const float *fx = s_fl + ( c & 1 )*10*NXF, *fy = fx + 5*NXF;
         if ( const int e = tid; e < NV2 )
         {
            const int i = e % NV, j = e / NV, p = ( j + 1 )*N + i + 1;
            float L[5], Rr[5], F[5];
#           pragma unroll
            for (int v=0; v<5; v++) { L[v] = w0[v*N2 + p];  Rr[v] = w1[v*N2 + p]; }
            hllc_pair_core<2,5>( ph, L, Rr, make_float2( w0[5*N2 + p], w1[5*N2 + p] ), make_float2( w0[6*N2 + p], w1[6*N2 + p] ),
                                 make_float2( w0[7*N2 + p], w1[7*N2 + p] ), F );
            bool nan = false;
#           pragma unroll
            for (int v=0; v<5; v++) nan |= ( F[v] != F[v] );
            if ( nan ) riemann_hlle_outlined<2,P,5>( ph, L, Rr, F );
            if ( c >= 1 )
            {
               float u[5], w[5];
#              pragma unroll
               for (int v=0; v<5; v++)
               {
                  const float *x = fx + v*NXF + j*NF + i, *y = fy + v*NXF + j*NV + i;
                  const A dfx = (A)x[1] - (A)x[0], dfy = (A)y[NV] - (A)y[0], dfz = (A)F[v] - (A)fzl[v];
                  u[v] = (float)( (A)L[v] - k2*( ( dfx + dfy ) + dfz ) );
               }
               u[0] = gmax( u[0], ph.min_dens );
               u[4] = floor_eint_in_engy<P>( ph, u[0], u[1], u[2], u[3], u[4] );
               con2pri_cc<P,5>( ph, u, w );
#              pragma unroll
               for (int v=0; v<5; v++) h[(size_t)v*NV3 + (size_t)( c - 1 )*NV2 + e] = w[v];
            }
#           pragma unroll
            for (int v=0; v<5; v++) fzl[v] = F[v];
         }
         if ( c < np ) faces( c + 1 );
         derive( c + 2, ( tid + nth - NXF % nth ) % nth );
         __syncthreads();
         if ( *s_abort )
         {
            if ( tid == 0 && c + 3 < nz ) mbar_wait_bounded( &bar[( c + 3 ) & 3], ( ( phase >> ( ( c + 3 ) & 3 ) ) + (uint32_t)( ( c + 3 ) >> 2 ) ) & 1u );
            __syncthreads();
            return;
         }
         if ( tid == 0 ) issue( c + 4 );           // the slot of plane c, last read in this step
      }
      for (int q=0; q<4; q++) phase ^= ( ( ( nz - q + 3 ) >> 2 ) & 1u ) << q;
      __syncthreads();
   }
}

// whole patch groups while they fill every slot, the rest in the slabs that need the fewest plane steps
template <typename R>
void rp_plan( RpArgs<R> &a, int slots, int nv )
{
   a.nitem = a.nwhole = a.npg;
   a.nslab = 1;
   const int rest = a.npg % slots;
   int best = nv + 3;
   for (int n : { 2, 4, 5, 10, 20, 11, 22 })
   {
      if ( rest == 0 || nv % n != 0 ) continue;
      const int steps = ( ( rest*n + slots - 1 )/slots )*( nv/n + 3 );
      if ( steps < best ) { best = steps;  a.nslab = n; }
   }
   if ( a.nslab == 1 ) return;
   a.nwhole = a.npg - rest;
   a.nitem  = a.nwhole + rest*a.nslab;
}

template <int P, int NXI>
cudaError_t rp_half_hllc_launch( RpArgs<float> a, cudaStream_t st )
{
   const void *fn = (const void*)rp_half_hllc_kernel<P,NXI>;
   constexpr int smem = RpxSmem<NXI>::bytes;
   int dev = 0, nsm = 0, per_sm = 0;
   cudaGetDevice( &dev );
   cudaDeviceGetAttribute( &nsm, cudaDevAttrMultiProcessorCount, dev );
   cudaError_t e = cudaFuncSetAttribute( fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem );
   if ( e == cudaSuccess ) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor( &per_sm, fn, RpxSmem<NXI>::THREADS, smem );
   if ( e != cudaSuccess ) return e;
   if ( per_sm < 1 ) return cudaErrorInvalidConfiguration;
   if ( a.npg == 0 ) return cudaSuccess;
   rp_plan( a, nsm*per_sm, NXI - 2 );
   const int grid = ( nsm*per_sm < a.nitem ) ? nsm*per_sm : a.nitem;
   rp_half_hllc_kernel<P,NXI><<< grid, RpxSmem<NXI>::THREADS, smem, st >>>( a );
   return cudaGetLastError();
}

// one launch over npg patch groups (persistent grid: SMs x resident CTAs)
template <typename R, int P, int RS, int NC, int NXI>
cudaError_t rp_half_launch( const RpArgs<R> &a, cudaStream_t st )
{
   const void *fn = (const void*)mhm_rp_half_kernel<R,P,RS,NC,NXI>;
   const size_t smem = rp_half_smem( sizeof(R), NC, NXI );
   int dev = 0, nsm = 0, per_sm = 0;
   cudaGetDevice( &dev );
   cudaDeviceGetAttribute( &nsm, cudaDevAttrMultiProcessorCount, dev );
   cudaError_t err = cudaFuncSetAttribute( fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem );
   if ( err != cudaSuccess ) return err;
   err = cudaOccupancyMaxActiveBlocksPerMultiprocessor( &per_sm, fn, RPH_BLOCK, smem );
   if ( err != cudaSuccess ) return err;
   if ( per_sm < 1 ) return cudaErrorInvalidConfiguration;
   int grid = nsm*per_sm;
   if ( grid > a.npg ) grid = a.npg;
   if ( grid == 0 ) return cudaSuccess;
   mhm_rp_half_kernel<R,P,RS,NC,NXI><<< grid, RPH_BLOCK, smem, st >>>( a );
   return cudaGetLastError();
}

template <typename R, int P, int NXI>
cudaError_t rp_half_pick_n( int rs, int nc, const RpArgs<R> &a, cudaStream_t st )
{
   if constexpr ( std::is_same<R, float>::value )
   {
      if ( rs == RS_HLLC && nc == 5 ) return rp_half_hllc_launch<P,NXI>( a, st );
   }
   else if ( rs == RS_HLLC && nc == 5 ) return rp_half_launch<R,P,RS_HLLC,5,NXI>( a, st );
   if ( rs == RS_HLLC && nc == 6 ) return rp_half_launch<R,P,RS_HLLC,6,NXI>( a, st );
   if ( rs == RS_HLLE && nc == 5 ) return rp_half_launch<R,P,RS_HLLE,5,NXI>( a, st );
   if ( rs == RS_HLLE && nc == 6 ) return rp_half_launch<R,P,RS_HLLE,6,NXI>( a, st );
   if ( rs == RS_ROE  && nc == 5 ) return rp_half_launch<R,P,RS_ROE,5,NXI>( a, st );
   if ( rs == RS_ROE  && nc == 6 ) return rp_half_launch<R,P,RS_ROE,6,NXI>( a, st );
   // two user passive scalars, without / with the dual-energy field (FP64 with 8 variables on the
   // 24^3 PPM input needs 237 KB of shared memory, above a CTA's 227 KB)
   if ( sizeof(R) == 8 && nc == 8 && NXI == 24 ) return cudaErrorNotSupported;
   if constexpr ( !( sizeof(R) == 8 && NXI == 24 ) )
   {
      if ( rs == RS_HLLC && nc == 8 ) return rp_half_launch<R,P,RS_HLLC,8,NXI>( a, st );
      if ( rs == RS_HLLE && nc == 8 ) return rp_half_launch<R,P,RS_HLLE,8,NXI>( a, st );
      if ( rs == RS_ROE  && nc == 8 ) return rp_half_launch<R,P,RS_ROE,8,NXI>( a, st );
   }
   if ( rs == RS_HLLC && nc == 7 ) return rp_half_launch<R,P,RS_HLLC,7,NXI>( a, st );
   if ( rs == RS_HLLE && nc == 7 ) return rp_half_launch<R,P,RS_HLLE,7,NXI>( a, st );
   if ( rs == RS_ROE  && nc == 7 ) return rp_half_launch<R,P,RS_ROE,7,NXI>( a, st );
   return cudaErrorNotSupported;
}

template <typename R, int P>
cudaError_t rp_half_pick( int rs, int nc, int nxi, const RpArgs<R> &a, cudaStream_t st )
{
   if ( nxi == 22 ) return rp_half_pick_n<R,P,22>( rs, nc, a, st );
   if ( nxi == 24 ) return rp_half_pick_n<R,P,24>( rs, nc, a, st );
   return cudaErrorNotSupported;
}

// The half step of npg patch groups: in [npg][nc][nxi^3] -> half [npg][nc][(nxi-2)^3] (nxi = FLU_NXT:
// 22 with PLM, 24 with PPM); ph carries the floors, the passive-floor mask and the reconstruction
// options.  Asynchronous on st.
int mhm_rp_half( int precision, int rsolver, int nc, int nxi, const void *in, void *half, int npg, double dt,
                 double dh, const Phys<double> &phd, int *status, cudaStream_t st )
{
   cudaError_t err;
   if ( precision == GB_PREC_FP64 )
   {
      RpArgs<double> a;
      memset( (void*)&a, 0, sizeof(a) );
      a.status = status;
      a.in = (const double*)in;  a.half = (double*)half;  a.npg = npg;
      a.dt_dh2 = 0.5*dt/dh;  a.ph = phd;
      err = rp_half_pick<double,P_FP64>( rsolver, nc, nxi, a, st );
   }
   else
   {
      RpArgs<float> a;
      memset( (void*)&a, 0, sizeof(a) );
      a.status = status;
      a.in = (const float*)in;  a.half = (float*)half;  a.npg = npg;
      a.dt_dh2 = (float)0.5f*(float)dt/(float)dh;
      a.ph.gamma = (float)phd.gamma;  a.ph.gm1 = (float)phd.gm1;  a.ph.inv_gm1 = (float)phd.inv_gm1;
      a.ph.min_dens = (float)phd.min_dens;  a.ph.min_pres = (float)phd.min_pres;  a.ph.min_eint = (float)phd.min_eint;
      a.ph.de_switch = (float)phd.de_switch;  a.ph.jeans_coeff = (float)phd.jeans_coeff;  a.ph.jeans = phd.jeans;
      a.ph.frac_mask = phd.frac_mask;  a.ph.pfloor = phd.pfloor;
      err = ( precision == GB_PREC_MIXED ) ? rp_half_pick<float,P_MIXED>( rsolver, nc, nxi, a, st )
                                           : rp_half_pick<float,P_FP32>( rsolver, nc, nxi, a, st );
   }
   if ( err == cudaErrorNotSupported ) return GB_E_UNSUPPORTED;
   return ( err == cudaSuccess ) ? GB_OK : GB_E_CUDA;
}

} // namespace gb
