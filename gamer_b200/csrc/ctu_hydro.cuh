// Hydro CTU: sizes, call parameters and the traced face values of a cell, shared by the separate
// kernels (ctu_hydro.cu) and the plane-streaming kernel (ctu_fused.cuh).
#pragma once
#include <cstring>
#include <type_traits>
#include "../../include/gamer_b200_fluid.h"
#include "hydro_physics.cuh"

namespace gb {

// generalized MinMod with theta < 2, which the plane-streaming kernel has built in
inline bool hctu_gmm( const gb_fluid_params &prm ) { return prm.lr_limiter == GB_LIM_GMINMOD && (float)prm.minmod_coeff < 2.0f; }

namespace hctu {
constexpr int NX  = 20;                // FLU_NXT
constexpr int NX3 = NX*NX*NX;
constexpr int NF  = 18;                // N_FC_VAR = N_HF_FLUX = N_FL_FLUX
constexpr int NF3 = NF*NF*NF;
// input sizes of the reconstruction LR: PLM FLU_NXT 20 (LR_GHOST_SIZE 1, FLU_GHOST_SIZE 2), PPM
// FLU_NXT 22 (2, 3) (include/Macro.h:643-665); the face-state, flux and output grids are the same
template <int LR> struct G {
   static constexpr int NX  = ( LR == LR_PPM ) ? 22 : 20;   // FLU_NXT
   static constexpr int NX3 = NX*NX*NX;
   static constexpr int LRG = ( LR == LR_PPM ) ? 2 : 1;     // LR_GHOST_SIZE
   static constexpr int FLG = LRG + 1;                       // FLU_GHOST_SIZE
};

GB_DEV int idx3( int i, int j, int k, int ni, int nj ) { return ( k*nj + j )*ni + i; }

template <typename R>
struct Args {
   const R *in;      // [npg][NC][20^3]
   R *out;           // [npg][NC][16^3]
   R *flux;          // [npg][9][NC][16^2]  (nullptr: not stored)
   char *de;         // [npg][16^3] dual-energy status (NC = 6 or 8; nullptr: not stored)
   R *pri;           // scratch [npg][NC][20^3]
   R *fcv;           // scratch [npg][6][NC][18^3]
   R *fcf;           // scratch [npg][3][NC][18^3]
   int npg, limiter;
   int nnorm;        // NormPassive: number of listed passive scalars (0 = off)
   int norm_idx[4];  // NormIdx (passive indices, no repeats)
   R coeff, dt, dh;
   Phys<R> ph;
};
}

// ---- PLM / PPM + characteristic tracing along D (CPU_Shared_DataReconstruction.cpp:376-560, hydro) ----
// RS: the HLL solvers trace with all waves (:454-477, HLL_INCLUDE_ALL_WAVES), so the sum over the waves
// m of R_m l_m( ev_m ) L_m d, with l_m linear (PLM) or quadratic (PPM) in the eigenvalue, is that
// polynomial of the primitive-variable Jacobian A applied to d: two to four sparse products with A
// (two non-zero terms a row) in place of the eigenvectors, their projections and the square root.
// Roe and the exact solver trace each face from the reference state of the fastest wave toward it
// (:513-553) with Hydro_GetEigenSystem's vectors (:1611-1892, no MHD): eigenvalues v_d - a, v_d (x3),
// v_d + a; the vectors in the rotated frame (rho, v_n, v_t1, v_t2, P) do not depend on the direction.
// CH: CHAR_RECONSTRUCTION, the slopes limited in the characteristic variables of the cell.
// LR_PPM: PPM face values (:704-1135, the limited slopes of the cell and its two neighbours, the
// parabola and its monotonicity constraint) and the tracing of the parabola (:1136-1290): each
// wave's correction over its domain of dependence adds the curvature term dfc6 = 6 (cc - (fL+fR)/2).
//
// The traced and floored primitive face values fl / fr of a cell cc with its neighbours along D at
// pl[v*st], pr[v*st] (PPM also two cells away, pll and prr).

// A d in the rotated frame (rho, v_n, v_t1, v_t2, P); gp = gamma P
template <typename R>
GB_DEV void hydro_jacobian( R vn, R rho, R irho, R gp, const R (&d)[5], R (&y)[5] )
{
   y[0] = vn*d[0] + rho*d[1];
   y[1] = vn*d[1] + irho*d[4];
   y[2] = vn*d[2];
   y[3] = vn*d[3];
   y[4] = vn*d[4] + gp*d[1];
}

template <int D, int RS, int NC, int CH, int LR, typename R>
GB_DEV void hctu_faces( const Phys<R> &ph, int limiter, R coeff, bool clamp, R dt_dh2, const R *pll, const R *pl, const R *cc,
                        const R *pr, const R *prr, int st, R (&fl)[NC], R (&fr)[NC] )
{
   typedef Dir<D> M;
   if constexpr ( LR == LR_PPM )
   {
      // the slopes of the cells c-1, c, c+1 (limited in primitive or characteristic variables)
      R sl[NC], sc[NC], sr[NC];
      if constexpr ( CH )
      {
         R ll[NC], cl[NC], cr[NC], rr[NC];
#        pragma unroll
         for (int v=0; v<NC; v++) { ll[v] = pll[v*st];  cl[v] = pl[v*st];  cr[v] = pr[v*st];  rr[v] = prr[v*st]; }
         ppm_char_slopes<D,NC>( ph, ll, cl, cc, cr, rr, limiter, coeff, sl, sc, sr );
      }
      else
      {
#        pragma unroll
         for (int v=0; v<NC; v++)
         {
            sl[v] = limit_slope( pll[v*st], pl[v*st], cc[v],     limiter, coeff );
            sc[v] = limit_slope( pl[v*st],  cc[v],    pr[v*st],  limiter, coeff );
            sr[v] = limit_slope( cc[v],     pr[v*st], prr[v*st], limiter, coeff );
         }
      }
#     pragma unroll
      for (int v=0; v<NC; v++) ppm_faces( pl[v*st], cc[v], pr[v*st], sl[v], sc[v], sr[v], limiter, fl[v], fr[v] );
   }
   else if constexpr ( CH )
   {
      R cl[NC], cr[NC];
#     pragma unroll
      for (int v=0; v<NC; v++) { cl[v] = pl[v*st];  cr[v] = pr[v*st]; }
      plm_faces_char<D,NC>( ph, cl, cc, cr, limiter, coeff, fl, fr );
   }
   else
   {
#     pragma unroll
      for (int v=0; v<NC; v++) plm_faces( pl[v*st], cc[v], pr[v*st], limiter, coeff, clamp, fl[v], fr[v] );
   }
   const R rho = cc[0], irho = R(1)/rho;
   const R a2 = ph.gamma*cc[4]/rho;
   const int wv[5] = { 0, M::n, M::t1, M::t2, 4 };
   R dfc[5], corl[5], corr[5];
#  pragma unroll
   for (int q=0; q<5; q++) dfc[q] = fr[wv[q]] - fl[wv[q]];
   if constexpr ( RS == RS_HLLC || RS == RS_HLLE )
   {
      // a sound speed that is zero, infinite or not a number leaves no eigenvectors: NaN face values,
      // as from the wave sums
      const R vn = ( a2 > R(0) && a2 <= Lim<R>::huge() ) ? cc[M::n] : R(NAN);
      const R gp = ph.gamma*cc[4];
      R y[5];
      if constexpr ( LR == LR_PPM )
      {
         R d6[5], e[5], y6[5], yy6[5];
#        pragma unroll
         for (int q=0; q<5; q++) d6[q] = R(6)*( cc[wv[q]] - R(0.5)*( fl[wv[q]] + fr[wv[q]] ) );
         hydro_jacobian( vn, rho, irho, gp, d6, y6 );
         hydro_jacobian( vn, rho, irho, gp, y6, yy6 );
         hydro_jacobian( vn, rho, irho, gp, dfc, e );
         const R c2 = R(4.0/3.0)*dt_dh2*dt_dh2;
#        pragma unroll
         for (int q=0; q<5; q++)
         {
            const R cur = -c2*yy6[q];
            corl[q] = cur - dt_dh2*( e[q] + y6[q] );
            corr[q] = cur - dt_dh2*( e[q] - y6[q] );
         }
      }
      else
      {
         hydro_jacobian( vn, rho, irho, gp, dfc, y );
#        pragma unroll
         for (int q=0; q<5; q++) corl[q] = corr[q] = -dt_dh2*y[q];
      }
   }
   else
   {
      const R as = gsqrt( a2 ), ia = R(1)/as, ia2 = ia*ia, vn = cc[M::n];
      R LE[5][5], RE[5][5];
#     pragma unroll
      for (int r=0; r<5; r++)
#        pragma unroll
         for (int q=0; q<5; q++) { LE[r][q] = R(0);  RE[r][q] = R(0); }
      LE[0][1] = -R(0.5)*rho*ia;  LE[0][4] = R(0.5)*ia2;
      LE[1][0] = R(1);            LE[1][4] = -ia2;
      LE[2][2] = R(1);            LE[3][3] = R(1);
      LE[4][1] = -LE[0][1];       LE[4][4] = LE[0][4];
      RE[0][0] = R(1);  RE[0][1] = -as*irho;  RE[0][4] = a2;
      RE[1][0] = R(1);
      RE[2][2] = R(1);  RE[3][3] = R(1);
      RE[4][0] = R(1);  RE[4][1] = -RE[0][1];  RE[4][4] = a2;
      const R ev[5] = { vn - as, vn, vn, vn, vn + as };
      // the reference states of the fastest waves, then the waves toward each face relative to them;
      // uncontracted, as the reference's CPU build: sums that cancel do so exactly
      const R cl0 = -dt_dh2*gmin( ev[0], R(0) ), cr0 = -dt_dh2*gmax( ev[4], R(0) );
      if constexpr ( LR == LR_PPM )
      {
         R dfc6[5];
#        pragma unroll
         for (int q=0; q<5; q++) dfc6[q] = R(6)*( cc[wv[q]] - R(0.5)*( fl[wv[q]] + fr[wv[q]] ) );
#        pragma unroll
         for (int q=0; q<5; q++)
         {
            corl[q] = cl0*( dfc[q] + ( R(1) - R(4.0/3.0)*cl0 )*dfc6[q] );
            corr[q] = cr0*( dfc[q] - ( R(1) + R(4.0/3.0)*cr0 )*dfc6[q] );
         }
#        pragma unroll
         for (int m=0; m<5; m++)
         {
            if ( ev[m] <= R(0) )
            {
               const R cC = dt_dh2*( ev[0] - ev[m] ), cD = R(4.0/3.0)*dt_dh2*cC*( ev[0] + ev[m] );
               R cf = R(0);
#              pragma unroll
               for (int q=0; q<5; q++) cf += LE[m][q]*( cC*( dfc[q] + dfc6[q] ) + cD*dfc6[q] );
#              pragma unroll
               for (int q=0; q<5; q++) corl[q] = corl[q] + mul_rn( cf, RE[m][q] );
            }
            if ( ev[m] >= R(0) )
            {
               const R cA = dt_dh2*( ev[4] - ev[m] ), cB = R(4.0/3.0)*dt_dh2*cA*( ev[4] + ev[m] );
               R cf = R(0);
#              pragma unroll
               for (int q=0; q<5; q++) cf += LE[m][q]*( cA*( dfc[q] - dfc6[q] ) + cB*dfc6[q] );
#              pragma unroll
               for (int q=0; q<5; q++) corr[q] = corr[q] + mul_rn( cf, RE[m][q] );
            }
         }
      }
      else
      {
#        pragma unroll
         for (int q=0; q<5; q++) { corl[q] = mul_rn( cl0, dfc[q] );  corr[q] = mul_rn( cr0, dfc[q] ); }
#        pragma unroll
         for (int m=0; m<5; m++)
         {
            if ( ev[m] <= R(0) )
            {
               R cf = R(0);
#              pragma unroll
               for (int q=0; q<5; q++) cf += LE[m][q]*dfc[q];
               cf *= dt_dh2*( ev[0] - ev[m] );
#              pragma unroll
               for (int q=0; q<5; q++) corl[q] = corl[q] + mul_rn( cf, RE[m][q] );
            }
            if ( ev[m] >= R(0) )
            {
               R cf = R(0);
#              pragma unroll
               for (int q=0; q<5; q++) cf += LE[m][q]*dfc[q];
               cf *= dt_dh2*( ev[4] - ev[m] );
#              pragma unroll
               for (int q=0; q<5; q++) corr[q] = corr[q] + mul_rn( cf, RE[m][q] );
            }
         }
      }
   }
   // passive scalars travel with the flow: the entropy wave only (:555-562); with PPM the parabola
   // integrated over its domain (:1262-1273)
   if constexpr ( NC > 5 )
   {
      const R cl = -dt_dh2*gmin( cc[M::n], R(0) ), cr = -dt_dh2*gmax( cc[M::n], R(0) );
#     pragma unroll
      for (int v=5; v<NC; v++)
      {
         const R dv = fr[v] - fl[v];
         if constexpr ( LR == LR_PPM )
         {
            const R dv6 = R(6)*( cc[v] - R(0.5)*( fl[v] + fr[v] ) );
            fl[v] += cl*( dv + ( R(1) - R(4.0/3.0)*cl )*dv6 );
            fr[v] += cr*( dv - ( R(1) + R(4.0/3.0)*cr )*dv6 );
         }
         else
         {
            fl[v] += cl*dv;
            fr[v] += cr*dv;
         }
      }
   }
#  pragma unroll
   for (int q=0; q<5; q++) { fl[wv[q]] += corl[q];  fr[wv[q]] += corr[q]; }
   fl[0] = gmax( fl[0], ph.min_dens );  fr[0] = gmax( fr[0], ph.min_dens );
   fl[4] = check_floor( fl[4], ph.min_pres );  fr[4] = check_floor( fr[4], ph.min_pres );
#  pragma unroll
   for (int v=5; v<NC; v++)
      if ( ph.pfloor & ( 1u << v ) ) { fl[v] = gmax( fl[v], Lim<R>::tiny() );  fr[v] = gmax( fr[v], Lim<R>::tiny() ); }
}

// the parameters of a call on n patch groups from number p0 on (without the scratch arrays)
template <typename R, int NC, int LR>
hctu::Args<R> hctu_args( const gb_fluid_config &cfg, const void *in, void *out, void *flux, char *de, int p0, int n,
                         const gb_fluid_params *prm )
{
   using namespace hctu;
   constexpr int NX3 = G<LR>::NX3;
   Args<R> a;
   memset( &a, 0, sizeof(a) );
   a.in   = (const R*)in  + (size_t)p0*NC*NX3;
   a.out  = (R*)out + (size_t)p0*NC*PS2*PS2*PS2;
   a.flux = ( prm->store_flux && flux ) ? (R*)flux + (size_t)p0*9*NC*PS2*PS2 : nullptr;
   a.de   = ( NC > 5 && de ) ? de + (size_t)p0*PS2*PS2*PS2 : nullptr;
   a.npg  = n;
   a.limiter = prm->lr_limiter;
   a.coeff = (R)prm->minmod_coeff;
   a.dt = (R)prm->dt;  a.dh = (R)prm->dh;
   a.ph.gamma = (R)cfg.gamma;  a.ph.gm1 = (R)( cfg.gamma - 1.0 );  a.ph.inv_gm1 = (R)( 1.0/( cfg.gamma - 1.0 ) );
   a.ph.min_dens = (R)prm->min_dens;  a.ph.min_pres = (R)prm->min_pres;  a.ph.min_eint = (R)prm->min_eint;
   a.ph.de_switch = (R)prm->dual_energy_switch;
   a.ph.jeans = prm->jeans_min_pres;  a.ph.jeans_coeff = (R)prm->jeans_min_pres_coeff;
   a.ph.pfloor = 0u;
   for (int v=5; v<NC; v++) if ( prm->passive_floor & ( 1LL << v ) ) a.ph.pfloor |= 1u << v;
   // FracPassive (mass fractions in the reconstruction) and NormPassive of the user scalars
   a.ph.frac_mask = 0u;
   if ( prm->frac_passive ) for (int k=0; k<prm->nfrac; k++) a.ph.frac_mask |= 1u << prm->frac_idx[k];
   a.nnorm = 0;
   if ( prm->norm_passive )
   {
      a.nnorm = prm->nnorm;
      for (int k=0; k<prm->nnorm && k<4; k++) a.norm_idx[k] = prm->norm_idx[k];
   }
   return a;
}

} // namespace gb
