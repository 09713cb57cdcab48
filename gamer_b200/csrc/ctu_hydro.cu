// Hydro CTU patch-group solver: PLM with characteristic tracing (HLL solvers: all waves,
// HLL_NO_REF_STATE; Roe and exact solvers: the reference states of the fastest waves), half-step
// Riemann fluxes, transverse-gradient correction, full-step Riemann fluxes, update.
//
// Reference path replaced: CPU_FluidSolver_CTU without MHD
// (src/Model_Hydro/CPU_Hydro/CPU_FluidSolver_CTU.cpp:157-342, Hydro_TGradientCorrection :368-599).
// Sizes (CTU, no MHD): PLM FLU_NXT 20, FLU_GHOST_SIZE 2, LR_GHOST_SIZE 1; PPM FLU_NXT 22, 3, 2;
// N_FC_VAR = N_HF_FLUX = N_FL_FLUX = 18 for both (include/CUFLU.h:107-118, include/Macro.h:643-665).
// Like the MHD pipeline, the stages are separate kernels over (patch group x cell/face) items with
// per-patch-group scratch (~1.2 MB in FP32), run over chunks of patch groups.
// Dual energy (DE_ENPY, NC = 6): the dual-energy field is the last variable, a passive scalar to the
// reconstruction (traced with the entropy wave, :555-562), the Riemann solvers (upwinded with the
// mass flux) and the transverse correction, floored by PassiveFloor, and the full step ends with the
// dual-energy fix of Hydro_FullStepUpdate (CPU_Shared_FullStepUpdate.cpp:144-201).
#include "ctu_hydro.cuh"

namespace gb {

// the plane-streaming kernel (ctu_fused.cuh), one instantiation unit per policy
int ctu_fused_fp32 ( const gb_fluid_config &cfg, const void *in, void *out, void *flux, int npg, const gb_fluid_params *prm, int *status, cudaStream_t st );
int ctu_fused_mixed( const gb_fluid_config &cfg, const void *in, void *out, void *flux, int npg, const gb_fluid_params *prm, int *status, cudaStream_t st );
int ctu_fused_fp64 ( const gb_fluid_config &cfg, const void *in, void *out, void *flux, int npg, const gb_fluid_params *prm, int *status, cudaStream_t st );

// items of one patch group per grid.z index (blockIdx.z = patch group of the chunk), 32-bit indices
#define HCTU_PG_LOOP( r, per ) \
   const int pg = blockIdx.z; \
   for (int r = blockIdx.x*blockDim.x + threadIdx.x; r < ( per ); r += gridDim.x*blockDim.x)

// kernels over the three face directions run them along grid.y, so that each direction's extents
// are compile-time constants (index decoding by constant division, no divergence)
#define HCTU_DIR( call ) \
   if      ( blockIdx.y == 0 ) { call( 0 ); } \
   else if ( blockIdx.y == 1 ) { call( 1 ); } \
   else                        { call( 2 ); }

// ---- conserved -> primitive (CPU_Shared_DataReconstruction.cpp:300-336) ----------------------
template <typename R, int P, int NC, int LR>
__global__ void hctu_con2pri( const __grid_constant__ hctu::Args<R> a )
{
   using namespace hctu;
   constexpr int NX3 = G<LR>::NX3;
   HCTU_PG_LOOP( c, NX3 )
   {
      const R *u = a.in + (size_t)pg*NC*NX3;
      R cu[NC], w[NC];
#     pragma unroll
      for (int v=0; v<NC; v++) cu[v] = u[v*NX3 + c];
      con2pri_cc<P,NC>( a.ph, cu, w );
      R *pri = a.pri + (size_t)pg*NC*NX3;
#     pragma unroll
      for (int v=0; v<NC; v++) pri[v*NX3 + c] = w[v];
   }
}

template <typename R, int P, int RS, int NC, int CH, int LR>
__global__ void __launch_bounds__( 256, ( sizeof(R) == 8 ) ? 1 : 4 ) hctu_recon( const __grid_constant__ hctu::Args<R> a )
{
   using namespace hctu;
   constexpr int NX = G<LR>::NX, NX3 = G<LR>::NX3, LRG = G<LR>::LRG;
   const int d = blockIdx.y;
   HCTU_PG_LOOP( f, NF3 )
   {
      const int ci = f % NF + LRG, cj = ( f / NF ) % NF + LRG, ck = f / ( NF*NF ) + LRG;
      const R *pri = a.pri + (size_t)pg*NC*NX3;
      const int c = idx3( ci, cj, ck, NX, NX );
      R cc[NC], fcon[2][NC];
#     pragma unroll
      for (int v=0; v<NC; v++) cc[v] = pri[v*NX3 + c];
      const R dt_dh2 = R(0.5)*a.dt/a.dh, *q = pri + c;
      R fl[NC], fr[NC];
      if      ( d == 0 ) hctu_faces<0,RS,NC,CH,LR>( a.ph, a.limiter, a.coeff, true, dt_dh2, q - 2, q - 1, cc, q + 1, q + 2, NX3, fl, fr );
      else if ( d == 1 ) hctu_faces<1,RS,NC,CH,LR>( a.ph, a.limiter, a.coeff, true, dt_dh2, q - 2*NX, q - NX, cc, q + NX, q + 2*NX, NX3, fl, fr );
      else               hctu_faces<2,RS,NC,CH,LR>( a.ph, a.limiter, a.coeff, true, dt_dh2, q - 2*NX*NX, q - NX*NX, cc, q + NX*NX, q + 2*NX*NX, NX3, fl, fr );
      pri2con<NC>( a.ph, fl, fcon[0] );
      pri2con<NC>( a.ph, fr, fcon[1] );
      R *fcv = a.fcv + (size_t)pg*6*NC*NF3;
#     pragma unroll
      for (int q=0; q<2; q++)
#        pragma unroll
         for (int v=0; v<NC; v++) fcv[( ( 2*d + q )*NC + v )*NF3 + f] = fcon[q][v];
   }
}

// ---- Riemann fluxes (Hydro_ComputeFlux, CPU_Shared_ComputeFlux.cpp:113-376) -------------------
// half step: NSkip_N = NSkip_T = 0 (17 x 18 x 18 faces per direction); full step: NSkip_N = 0,
// NSkip_T = 1 (17 x 16 x 16), with the coarse-fine planes (Hydro_StoreIntFlux :391-450, no MHD)
template <int D, typename R, int P, int RS, int FULL, int NC>
GB_DEV void hctu_face( const hctu::Args<R> &a, int pg, int fi, int fj, int fk )
{
   using namespace hctu;
   constexpr int st = FULL ? 1 : 0;                       // transverse skip
   const int sk[3] = { D == 0 ? 0 : st, D == 1 ? 0 : st, D == 2 ? 0 : st };
   const int dfc[3] = { 1, NF, NF*NF };
   const int ifc = idx3( fi + sk[0], fj + sk[1], fk + sk[2], NF, NF );
   const R *fcv = a.fcv + (size_t)pg*6*NC*NF3;
   R L[NC], Rr[NC], F[NC];
#  pragma unroll
   for (int v=0; v<NC; v++) { L[v] = fcv[( ( 2*D + 1 )*NC + v )*NF3 + ifc];  Rr[v] = fcv[( 2*D*NC + v )*NF3 + ifc + dfc[D]]; }
   riemann<RS,D,P,NC>( a.ph, L, Rr, F );
   R *fcf = a.fcf + (size_t)pg*3*NC*NF3;
   const int ix = idx3( fi, fj, fk, NF, NF );
#  pragma unroll
   for (int v=0; v<NC; v++) fcf[( D*NC + v )*NF3 + ix] = F[v];
   if ( FULL && a.flux != nullptr )
   {
      const int fl[3] = { fi, fj, fk };
      const int nrm = fl[D];
      if ( ( nrm & 7 ) == 0 )
      {
         // transverse index with the smaller axis number is the fastest
         const int a0 = ( D == 0 ) ? fj : fi, a1 = ( D == 2 ) ? fj : fk;
         R *dst = a.flux + (size_t)pg*9*NC*PS2*PS2 + (size_t)( 3*D + nrm/PS1 )*NC*PS2*PS2 + a1*PS2 + a0;
#        pragma unroll
         for (int v=0; v<NC; v++) dst[v*PS2*PS2] = F[v];
      }
   }
}

template <typename R, int P, int RS, int FULL, int NC>
__global__ void __launch_bounds__( 256, ( sizeof(R) == 8 ) ? 1 : 3 ) hctu_flux( const __grid_constant__ hctu::Args<R> a )
{
   using namespace hctu;
   constexpr int nn = NF - 1, nt = FULL ? NF - 2 : NF;         // faces along / across the normal
   constexpr int per = nn*nt*nt;
   HCTU_PG_LOOP( q, per )
   {
#     define HCTU_FACE( D ) { \
         constexpr int e0 = ( D == 0 ) ? nn : nt, e1 = ( D == 1 ) ? nn : nt; \
         hctu_face<D,R,P,RS,FULL,NC>( a, pg, q % e0, ( q / e0 ) % e1, q / ( e0*e1 ) ); }
      HCTU_DIR( HCTU_FACE )
#     undef HCTU_FACE
   }
}

// ---- transverse-gradient correction (Hydro_TGradientCorrection, CPU_FluidSolver_CTU.cpp:368-599,
// no MHD): along D the face cells of the whole 18-wide range, across it the inner 16 ----------------
template <int D, typename R, int P, int NC>
GB_DEV void hctu_tgrad_dir( const hctu::Args<R> &a, int pg, int i0, int j0, int k0 )
{
   using namespace hctu;
   constexpr int T1 = ( D + 1 ) % 3, T2 = ( D + 2 ) % 3;
   const int dfl[3] = { 1, NF, NF*NF };
   const int f = idx3( i0 + ( D != 0 ), j0 + ( D != 1 ), k0 + ( D != 2 ), NF, NF );
   R *fcv = a.fcv + (size_t)pg*6*NC*NF3;
   const R *F = a.fcf + (size_t)pg*3*NC*NF3;
   const R dt_dh2 = R(0.5)*a.dt/a.dh;
   R q0[NC], q1[NC];
#  pragma unroll
   for (int v=0; v<NC; v++) { q0[v] = fcv[( 2*D*NC + v )*NF3 + f];  q1[v] = fcv[( ( 2*D + 1 )*NC + v )*NF3 + f]; }
#  pragma unroll
   for (int v=0; v<NC; v++)
   {
      const R tg1 = F[( T1*NC + v )*NF3 + f] - F[( T1*NC + v )*NF3 + f - dfl[T1]];
      const R tg2 = F[( T2*NC + v )*NF3 + f] - F[( T2*NC + v )*NF3 + f - dfl[T2]];
      const R c = -dt_dh2*( tg1 + tg2 );
      q0[v] += c;  q1[v] += c;
   }
   q0[0] = gmax( q0[0], a.ph.min_dens );  q1[0] = gmax( q1[0], a.ph.min_dens );
   q0[4] = floor_eint_in_engy<P>( a.ph, q0[0], q0[1], q0[2], q0[3], q0[4] );
   q1[4] = floor_eint_in_engy<P>( a.ph, q1[0], q1[1], q1[2], q1[3], q1[4] );
#  pragma unroll
   for (int v=5; v<NC; v++)
      if ( a.ph.pfloor & ( 1u << v ) ) { q0[v] = gmax( q0[v], Lim<R>::tiny() );  q1[v] = gmax( q1[v], Lim<R>::tiny() ); }
#  pragma unroll
   for (int v=0; v<NC; v++) { fcv[( 2*D*NC + v )*NF3 + f] = q0[v];  fcv[( ( 2*D + 1 )*NC + v )*NF3 + f] = q1[v]; }
}

template <typename R, int P, int NC>
__global__ void hctu_tgrad( const __grid_constant__ hctu::Args<R> a )
{
   using namespace hctu;
   constexpr int N3 = NF*( NF - 2 )*( NF - 2 );
   HCTU_PG_LOOP( q, N3 )
   {
      // extent NF along d, NF-2 across
#     define HCTU_TG( D ) { \
         constexpr int e0 = ( D == 0 ) ? NF : NF - 2, e1 = ( D == 1 ) ? NF : NF - 2; \
         hctu_tgrad_dir<D,R,P,NC>( a, pg, q % e0, ( q / e0 ) % e1, q / ( e0*e1 ) ); }
      HCTU_DIR( HCTU_TG )
#     undef HCTU_TG
   }
}

// ---- full-step update (Hydro_FullStepUpdate, CPU_Shared_FullStepUpdate.cpp:64-271, no MHD) -------
template <typename R, int P, int NC, int LR>
__global__ void hctu_update( const __grid_constant__ hctu::Args<R> a )
{
   using namespace hctu;
   constexpr int NX = G<LR>::NX, NX3 = G<LR>::NX3, FLG = G<LR>::FLG;
   typedef typename std::conditional<P == P_MIXED, double, R>::type A;
   constexpr int N3 = PS2*PS2*PS2;
   const A dt_dh = (A)a.dt/(A)a.dh;
   HCTU_PG_LOOP( q, N3 )
   {
      const int io = q % PS2, jo = ( q / PS2 ) % PS2, ko = q / ( PS2*PS2 );
      const int ifl = idx3( io, jo, ko, NF, NF );
      const int dfl[3] = { 1, NF, NF*NF };
      const int iin = idx3( io + FLG, jo + FLG, ko + FLG, NX, NX );
      const R *F = a.fcf + (size_t)pg*3*NC*NF3;
      const R *u = a.in + (size_t)pg*NC*NX3;
      R *out = a.out + (size_t)pg*NC*N3;
      R w[NC];
#     pragma unroll
      for (int v=0; v<NC; v++)
      {
         A df[3];
#        pragma unroll
         for (int d=0; d<3; d++) df[d] = (A)F[( d*NC + v )*NF3 + ifl + dfl[d]] - (A)F[( d*NC + v )*NF3 + ifl];
         w[v] = (R)( (A)u[v*NX3 + iin] - dt_dh*( df[0] + df[1] + df[2] ) );
      }
      if constexpr ( NC > 5 )
      {
         // passive floor and normalisation, then the dual-energy fix (CPU_Shared_FullStepUpdate.cpp:144-201);
         // the dual-energy field is the last variable (NC = 6: alone, NC = 8: after two user scalars)
         constexpr bool DUAL = ( NC == 6 || NC == 8 );
         constexpr int  NPU  = NC - 5 - ( DUAL ? 1 : 0 );
#        pragma unroll
         for (int v=5; v<NC; v++) if ( a.ph.pfloor & ( 1u << v ) ) w[v] = gmax( w[v], Lim<R>::tiny() );
         if constexpr ( NPU > 0 ) if ( a.nnorm > 0 ) normalize_passive<NC>( w[0], w, a.nnorm, a.norm_idx );
         if constexpr ( DUAL )
         {
            const R ekin = R(0.5)*( w[1]*w[1] + w[2]*w[2] + w[3]*w[3] )/w[0];
            if ( w[0] > R(0) && w[4]*R(2) > ekin )
            {
               char st;
               dual_energy_fix<P>( a.ph, w[0], w[1], w[2], w[3], w[4], w[NC-1], st );
               if ( a.de != nullptr ) a.de[(size_t)pg*N3 + q] = st;
            }
         }
      }
#     pragma unroll
      for (int v=0; v<NC; v++) out[v*N3 + q] = w[v];
   }
}

// Whether a call of npg patch groups runs through the plane-streaming kernel (ctu_fused.cuh): five
// variables, limiting in primitive variables, HLLC or HLLE, and PLM, or PPM in FP32.
// It takes one time T per wave of patch groups (two CTAs per SM for PLM in float, one otherwise), 19
// dependent steps long, while the separate kernels spread any number over the whole GPU and take a time t
// per patch group: the line lies at npg = T/t per wave, with T from the slowest of a lognormal, a
// Kelvin-Helmholtz and a blast flow, for generalized MinMod with theta < 2 (built in) and for the other
// limiters (chosen at run time).  Measured on B200, us, streaming / separate:
//    FP32 PLM        MinMod 100 patch groups 122 / 127, 40: 123 / 60, 592: 312 / 653; others (van Albada)
//                    125: 164 / 165, 290: 204 / 354, but 297 to 310 a few us more than the separate ones
//    FP32 PPM HLLC   MinMod 100: 181 / 181, 592: 706 / 981; others 125: 261 / 248, 290: 515 / 551
//    FP32 PPM HLLE   MinMod 100: 192 / 179, 120: 193 / 217, 592: 756 / 979; others no gain (1000: 1850 / 1795)
//    mixed PLM       MinMod T 236 lognormal, 263 blast, t 1.08 (592: 474 / 664); others no gain (blast 580: 769 / 678)
//    FP64 PLM        MinMod 100: 210 / 232, 592: 834 / 1190; others 290: 565 / 646, blast 1000: 2154 / 2113
// Not built, since no line holds for every flow: Roe (its reference states lengthen the chain; lognormal
// FP32 592: 847 / 797, mixed 1334 / 978, FP64 1848 / 1662; Kelvin-Helmholtz 616 / 740, 756 / 752, 1361 / 1481),
// and PPM in mixed (one CTA per SM; 2000: 3381 / 3233, blast 1000: 1939 / 1638, Kelvin-Helmholtz 1068 / 1469).
// PPM in FP64 would need 266 KB of shared memory.
bool ctu_hydro_fused( const gb_fluid_config &cfg, const gb_fluid_params &prm, int npg )
{
   const bool ppm = ( cfg.lr_scheme == GB_LR_PPM ), hlle = ( cfg.rsolver == GB_RSOLVER_HLLE ), gmm = hctu_gmm( prm );
   if ( cfg.dual_energy != GB_DE_NONE || cfg.npassive_user != 0 || cfg.char_reconstruction ) return false;
   if ( ( cfg.rsolver != GB_RSOLVER_HLLC && !hlle ) || ( ppm && cfg.precision != GB_PREC_FP32 ) ) return false;
   int line;
   if      ( cfg.precision == GB_PREC_MIXED ) { if ( !gmm ) return false;  line = 245; }
   else if ( cfg.precision == GB_PREC_FP64 )  line = gmm ? 100 : 144;
   else if ( ppm && hlle )                    { if ( !gmm ) return false;  line = 110; }
   else if ( ppm )                            line = gmm ? 105 : 140;
   else                                       line = gmm ? 100 : 155;
   int dev = 0, nsm = 148;
   cudaGetDevice( &dev );
   cudaDeviceGetAttribute( &nsm, cudaDevAttrMultiProcessorCount, dev );
   const int slots = nsm*( ( ppm || cfg.precision == GB_PREC_FP64 ) ? 1 : 2 ), waves = ( npg + slots - 1 )/slots;
   return npg > 0 && npg >= line*waves;
}

namespace {

size_t hctu_scratch_per_pg( size_t rsz, int nc, int lr )
{
   using namespace hctu;
   const size_t nx3 = ( lr == LR_PPM ) ? G<LR_PPM>::NX3 : G<LR_PLM>::NX3;
   return rsz*( (size_t)nc*nx3 + 6*(size_t)nc*NF3 + 3*(size_t)nc*NF3 ) + 3*256;
}

// items of one patch group (and direction) along x, about 4 per thread; face directions along y;
// patch groups along z (the directions of one patch group are scheduled together, sharing L2)
dim3 hctu_grid( int per, int npg, int block, int ndir = 1 )
{
   return dim3( ( per + 4*block - 1 )/( 4*block ), ndir, npg );
}

template <typename R, int P, int RS, int NC, int LR>
int hctu_solve_t( const gb_fluid_config &cfg, const void *in, void *out, void *flux, char *de, int npg,
                  const gb_fluid_params *prm, void *scratch, size_t scratch_bytes, cudaStream_t st )
{
   using namespace hctu;
   constexpr int NX3 = G<LR>::NX3;
   size_t fit = scratch_bytes / hctu_scratch_per_pg( sizeof(R), NC, LR );
   if ( fit < 1 ) return GB_E_INVALID;
   const int chunk = ( fit > 65535 ) ? 65535 : (int)fit;
   for (int p0 = 0; p0 < npg; p0 += chunk)
   {
      const int n = ( npg - p0 < chunk ) ? npg - p0 : chunk;
      char *w = (char*)scratch;
      auto take = [&]( size_t elems ) { R *r = (R*)w;  w += ( elems*sizeof(R) + 255 ) & ~(size_t)255;  return r; };
      Args<R> a = hctu_args<R,NC,LR>( cfg, in, out, flux, de, p0, n, prm );
      a.pri  = take( (size_t)n*NC*NX3 );
      a.fcv  = take( (size_t)n*6*NC*NF3 );
      a.fcf  = take( (size_t)n*3*NC*NF3 );
      const int B = 256;
      hctu_con2pri<R,P,NC,LR><<< hctu_grid( NX3, n, B ), B, 0, st >>>( a );
      if ( cfg.char_reconstruction ) hctu_recon<R,P,RS,NC,1,LR><<< hctu_grid( NF3, n, B, 3 ), B, 0, st >>>( a );
      else                           hctu_recon<R,P,RS,NC,0,LR><<< hctu_grid( NF3, n, B, 3 ), B, 0, st >>>( a );
      hctu_flux<R,P,RS,0,NC><<< hctu_grid( ( NF - 1 )*NF*NF, n, B, 3 ), B, 0, st >>>( a );
      hctu_tgrad<R,P,NC><<< hctu_grid( NF*( NF - 2 )*( NF - 2 ), n, B, 3 ), B, 0, st >>>( a );
      hctu_flux<R,P,RS,1,NC><<< hctu_grid( ( NF - 1 )*( NF - 2 )*( NF - 2 ), n, B, 3 ), B, 0, st >>>( a );
      hctu_update<R,P,NC,LR><<< hctu_grid( PS2*PS2*PS2, n, B ), B, 0, st >>>( a );
      if ( cudaGetLastError() != cudaSuccess ) return GB_E_CUDA;
   }
   return GB_OK;
}

template <typename R, int P, int NC, int LR>
int hctu_solve_rs( const gb_fluid_config &cfg, const void *in, void *out, void *flux, char *de, int npg,
                   const gb_fluid_params *prm, void *scratch, size_t scratch_bytes, cudaStream_t st )
{
   if ( cfg.rsolver == GB_RSOLVER_HLLE )
      return hctu_solve_t<R,P,RS_HLLE,NC,LR>( cfg, in, out, flux, de, npg, prm, scratch, scratch_bytes, st );
   if ( cfg.rsolver == GB_RSOLVER_ROE )
      return hctu_solve_t<R,P,RS_ROE,NC,LR>( cfg, in, out, flux, de, npg, prm, scratch, scratch_bytes, st );
   if ( cfg.rsolver == GB_RSOLVER_EXACT )
      return hctu_solve_t<R,P,RS_EXACT,NC,LR>( cfg, in, out, flux, de, npg, prm, scratch, scratch_bytes, st );
   return hctu_solve_t<R,P,RS_HLLC,NC,LR>( cfg, in, out, flux, de, npg, prm, scratch, scratch_bytes, st );
}

template <typename R, int P, int LR>
int hctu_solve_nc( const gb_fluid_config &cfg, const void *in, void *out, void *flux, char *de, int npg,
                   const gb_fluid_params *prm, void *scratch, size_t scratch_bytes, cudaStream_t st )
{
   const bool dual = ( cfg.dual_energy == GB_DE_ENPY );
   if ( cfg.npassive_user == GB_NPASSIVE_USER )
   {
      static_assert( GB_NPASSIVE_USER == 2, "the passive-scalar instantiations are built for two user scalars" );
      return dual ? hctu_solve_rs<R,P,8,LR>( cfg, in, out, flux, de, npg, prm, scratch, scratch_bytes, st )
                  : hctu_solve_rs<R,P,7,LR>( cfg, in, out, flux, de, npg, prm, scratch, scratch_bytes, st );
   }
   if ( dual )
      return hctu_solve_rs<R,P,6,LR>( cfg, in, out, flux, de, npg, prm, scratch, scratch_bytes, st );
   return hctu_solve_rs<R,P,5,LR>( cfg, in, out, flux, de, npg, prm, scratch, scratch_bytes, st );
}

template <typename R, int P>
int hctu_solve_lr( const gb_fluid_config &cfg, const void *in, void *out, void *flux, char *de, int npg,
                   const gb_fluid_params *prm, void *scratch, size_t scratch_bytes, cudaStream_t st )
{
   if ( cfg.lr_scheme == GB_LR_PPM )
      return hctu_solve_nc<R,P,LR_PPM>( cfg, in, out, flux, de, npg, prm, scratch, scratch_bytes, st );
   return hctu_solve_nc<R,P,LR_PLM>( cfg, in, out, flux, de, npg, prm, scratch, scratch_bytes, st );
}

} // namespace

size_t ctu_hydro_scratch_bytes_per_pg( int precision, int ncomp, int lr_scheme )
{
   return hctu_scratch_per_pg( ( precision == GB_PREC_FP64 ) ? 8 : 4, ncomp, lr_scheme );
}

// one hydro CTU solve of npg patch groups: by the plane-streaming kernel (fused: ctu_hydro_fused of the
// caller's whole call, of which these may be a chunk), or by the separate kernels in chunks of
// scratch_bytes / ctu_hydro_scratch_bytes_per_pg
int ctu_hydro_solve( const gb_fluid_config &cfg, bool fused, const void *flu_in, void *flu_out, void *flux, char *de, int npg,
                     const gb_fluid_params *prm, void *scratch, size_t scratch_bytes, int *status, cudaStream_t st )
{
   if ( fused )
   {
      if ( cfg.precision == GB_PREC_FP64 )  return ctu_fused_fp64 ( cfg, flu_in, flu_out, flux, npg, prm, status, st );
      if ( cfg.precision == GB_PREC_MIXED ) return ctu_fused_mixed( cfg, flu_in, flu_out, flux, npg, prm, status, st );
      return ctu_fused_fp32( cfg, flu_in, flu_out, flux, npg, prm, status, st );
   }
   if ( cfg.precision == GB_PREC_FP64 )
      return hctu_solve_lr<double,P_FP64>( cfg, flu_in, flu_out, flux, de, npg, prm, scratch, scratch_bytes, st );
   if ( cfg.precision == GB_PREC_MIXED )
      return hctu_solve_lr<float,P_MIXED>( cfg, flu_in, flu_out, flux, de, npg, prm, scratch, scratch_bytes, st );
   return hctu_solve_lr<float,P_FP32>( cfg, flu_in, flu_out, flux, de, npg, prm, scratch, scratch_bytes, st );
}

} // namespace gb

extern "C" int gb_fluid_ctu_one_kernel( const gb_fluid_config *cfg, const gb_fluid_params *prm, int npg, int *one )
{
   if ( cfg == nullptr || prm == nullptr || one == nullptr || npg < 0 ) return GB_E_INVALID;
   *one = ( cfg->scheme == GB_SCHEME_CTU && cfg->rsolver != GB_RSOLVER_HLLD && gb::ctu_hydro_fused( *cfg, *prm, npg ) ) ? 1 : 0;
   return GB_OK;
}
