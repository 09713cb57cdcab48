// Coarse-to-fine spatial interpolation of GAMER's AMR ghost-zone fill and refinement
// (Interpolate(), src/Interpolation/Interpolate.cpp:90-206, and its schemes Int_*.cpp), for a batch
// of independent interpolation regions of one shape, and the window assembly of the ghost-zone fill.
//
// The reference interpolates a region dimension by dimension: the x pass turns every coarse line of
// the region (plus CGhost layers in y and z) into pairs of fine values, the y pass does the same on
// the x-pass result, the z pass on the y-pass result, each pass into a temporary array.  A fine cell
// of coarse parent (i,j,k) therefore depends only on the (2*CGhost+1)^3 coarse cells around it, so here
// one thread owns one coarse cell and produces its 2x2x2 fine children directly: the x operator on
// the (2G+1)^2 lines through the neighbourhood, the y operator on their results, the z operator last
// -- the same operands and the same operations as the reference's passes, with no temporary arrays.
// INT_MINMOD1D (unsplit) takes the three limited slopes of the parent directly.
//
// Interpolate_Iterate (:208-560), the path GAMER's hydro ghost-zone fill takes for the conserved
// variables (src/Main/InterpolateGhostZone.cpp:1805), is built too: a parent whose eight children
// include an unphysical state (Hydro_IsUnphysical) is interpolated again, first in primitive variables
// (OPT__INT_PRIM), then with the monotonicity coefficient reduced MONO_MAX_ITER times; with the
// reference's INTERP_MASK (include/Macro.h:947) every parent iterates on its own, so this is again one
// thread per parent.  A parent still failing after the last iteration sets GB_INTERP_FAILED (the
// reference aborts the run there).
//
// Every multiplication, addition and division is written with explicitly rounded intrinsics, so the
// compiler contracts nothing into FMA and divides are IEEE: the results equal the reference CPU build
// bit for bit (in FP64 always; in FP32 as long as no intermediate is subnormal -- the device flushes
// those to zero).
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>
#include "../../include/gamer_b200_fluid.h"
#include "gb_common.cuh"

namespace gb {
namespace {

// IntScheme_t (include/Typedef.h:171-180)
constexpr int INT_MINMOD3D = 1, INT_MINMOD1D = 2, INT_VANLEER = 3, INT_CQUAD = 4, INT_QUAD = 5, INT_CQUAR = 6,
              INT_QUAR = 7;

__host__ __device__ constexpr int int_ghost( int sch ) { return ( sch == INT_CQUAR || sch == INT_QUAR ) ? 2 : 1; }

// explicitly rounded arithmetic (never contracted into FMA)
GB_DEV float  radd( float a, float b )   { return __fadd_rn( a, b ); }
GB_DEV double radd( double a, double b ) { return __dadd_rn( a, b ); }
GB_DEV float  rsub( float a, float b )   { return __fsub_rn( a, b ); }
GB_DEV double rsub( double a, double b ) { return __dsub_rn( a, b ); }
GB_DEV float  rmul( float a, float b )   { return __fmul_rn( a, b ); }
GB_DEV double rmul( double a, double b ) { return __dmul_rn( a, b ); }
GB_DEV float  rdiv( float a, float b )   { return __fdiv_rn( a, b ); }
GB_DEV double rdiv( double a, double b ) { return __ddiv_rn( a, b ); }
GB_DEV float  rmin( float a, float b )   { return fminf( a, b ); }
GB_DEV double rmin( double a, double b ) { return fmin( a, b ); }
GB_DEV float  rmax( float a, float b )   { return fmaxf( a, b ); }
GB_DEV double rmax( double a, double b ) { return fmax( a, b ); }
GB_DEV float  rabs( float a )            { return fabsf( a ); }
GB_DEV double rabs( double a )           { return fabs( a ); }

template <typename R> GB_DEV R sign_of( R a ) { return ( a < R(0) ) ? R(-1) : R(+1); }   // SIGN (include/Macro.h:1178)

// the limited-slope fallback shared by the quadratic and quartic schemes: the centred slope
// 0.125*(R1 - L1) bounded by MonoCoeff/4 of each one-sided slope (Int_Quadratic.cpp, Int_Quartic.cpp)
template <typename R>
GB_DEV R mono_fallback( R L1, R R1, R ls, R rs, R mc4 )
{
   R s = rmul( R(0.125), rsub( R1, L1 ) );
   ls = rmul( ls, mc4 );
   rs = rmul( rs, mc4 );
   const R sg = sign_of( ls );
   s = rmul( s, sg );
   s = rmin( rmul( sg, ls ), s );
   s = rmin( rmul( sg, rs ), s );
   return rmul( s, sg );
}

// the conservative schemes' limiter on the half slope s (Int_CQuadratic.cpp, Int_CQuartic.cpp)
template <typename R>
GB_DEV R mono_conservative( R s, R ls, R rs, R coeff )
{
   const R sg = sign_of( ls );
   s  = rmul( s, sg );
   ls = rmul( ls, sg );
   rs = rmul( rs, sg );
   if ( ls < rs ) ls = rmul( ls, coeff );
   else           rs = rmul( rs, coeff );
   s = rmin( ls, s );
   s = rmin( rs, s );
   return rmul( s, sg );
}

// One dimension of a split scheme: the two fine children (lo, hi) of the centre c[G] of a line of
// 2G+1 coarse values.  coeff = the monotonicity coefficient of this iteration.
template <int SCH, typename R>
GB_DEV void op1d( const R *c, bool mono, R coeff, bool opp, R &lo, R &hi )
{
   constexpr int G = int_ghost( SCH );
   const R C = c[G], L1 = c[G-1], R1 = c[G+1];
   const bool flat = opp && rmul( L1, R1 ) < R(0);     // OppSign0thOrder
   if constexpr ( SCH == INT_MINMOD3D || SCH == INT_VANLEER )
   {
      const R ls = rsub( C, L1 ), rs = rsub( R1, C );
      R s;
      if ( rmul( rs, ls ) <= R(0) ) s = R(0);
      else if constexpr ( SCH == INT_MINMOD3D ) s = rmul( R(0.25), ( rabs( rs ) < rabs( ls ) ) ? rs : ls );
      else                                      s = rdiv( rmul( rmul( R(0.5), ls ), rs ), radd( ls, rs ) );
      if ( flat ) s = R(0);
      lo = rsub( C, s );  hi = radd( C, s );
   }
   else if constexpr ( SCH == INT_CQUAD || SCH == INT_CQUAR )
   {
      R s;
      if constexpr ( SCH == INT_CQUAD ) s = rmul( R(0.125), rsub( R1, L1 ) );
      else
      {
         const R L2 = c[0], R2 = c[4];
         s = radd( radd( radd( rmul( R(+3.0/128.0), L2 ), rmul( R(-22.0/128.0), L1 ) ), rmul( R(+22.0/128.0), R1 ) ),
                   rmul( R(-3.0/128.0), R2 ) );
      }
      if ( mono )
      {
         const R ls = rmul( R(0.25), rsub( C, L1 ) ), rs = rmul( R(0.25), rsub( R1, C ) );
         if ( rmul( ls, rs ) > R(0) )
         {
            if constexpr ( SCH == INT_CQUAR ) if ( rmul( s, ls ) < R(0) ) s = rmul( R(0.125), rsub( R1, L1 ) );
            s = mono_conservative( s, ls, rs, coeff );
         }
         else s = R(0);
      }
      if ( flat ) s = R(0);
      lo = rsub( C, s );  hi = radd( C, s );
   }
   else   // INT_QUAD / INT_QUAR: fixed-weight interpolation, limited where it over- or undershoots
   {
      if constexpr ( SCH == INT_QUAD )
      {
         lo = radd( radd( rmul( R(+5.0/32.0), L1 ), rmul( R(+30.0/32.0), C ) ), rmul( R(-3.0/32.0), R1 ) );
         hi = radd( radd( rmul( R(-3.0/32.0), L1 ), rmul( R(+30.0/32.0), C ) ), rmul( R(+5.0/32.0), R1 ) );
      }
      else
      {
         const R L2 = c[0], R2 = c[4];
         lo = radd( radd( radd( radd( rmul( R(-45.0/2048.0), L2 ), rmul( R(+420.0/2048.0), L1 ) ),
                                rmul( R(+1890.0/2048.0), C ) ), rmul( R(-252.0/2048.0), R1 ) ), rmul( R(+35.0/2048.0), R2 ) );
         hi = radd( radd( radd( radd( rmul( R(+35.0/2048.0), L2 ), rmul( R(-252.0/2048.0), L1 ) ),
                                rmul( R(+1890.0/2048.0), C ) ), rmul( R(+420.0/2048.0), R1 ) ), rmul( R(-45.0/2048.0), R2 ) );
      }
      if ( mono )
      {
         const R ls = rsub( C, L1 ), rs = rsub( R1, C );
         if ( rmul( ls, rs ) > R(0) )
         {
            const R cmax = ( ls > R(0) ) ? R1 : L1, cmin = ( ls > R(0) ) ? L1 : R1;
            bool over = rmax( lo, hi ) > cmax || rmin( lo, hi ) < cmin;
            if constexpr ( SCH == INT_QUAR ) over = over || rmul( rsub( hi, lo ), ls ) < R(0);
            if ( over )
            {
               const R s = mono_fallback( L1, R1, ls, rs, rmul( R(0.25), coeff ) );
               lo = rsub( C, s );  hi = radd( C, s );
            }
         }
         else { lo = C;  hi = C; }
      }
      if ( flat ) { lo = C;  hi = C; }
   }
}

// MinMod-1D limited slope of one direction (Int_MinMod1D.cpp)
template <typename R>
GB_DEV R minmod_slope( R L1, R C, R R1, bool opp )
{
   const R ls = rsub( C, L1 ), rs = rsub( R1, C );
   R s = ( rmul( rs, ls ) <= R(0) ) ? R(0) : rmul( R(0.25), ( rabs( rs ) < rabs( ls ) ) ? rs : ls );
   if ( opp && rmul( L1, R1 ) < R(0) ) s = R(0);
   return s;
}

template <typename R>
struct IntArgs {
   const R *cdata;            // [nbatch][ncomp][cz][cy][cx]
   R       *fdata;            // [nbatch][ncomp][fz][fy][fx]
   int      csize[3], cstart[3], crange[3], fsize[3], fstart[3];
   int      ncomp, nbatch;
   unsigned mono;             // bit v: Monotonic[v]
   R        mono_coeff;       // INT_MONO_COEFF
   int      opp;              // OppSign0thOrder
   // Interpolate_Iterate (hydro conserved variables, ncomp = 5)
   int      int_prim;         // OPT__INT_PRIM: second attempt in primitive variables
   int      mono_max_iter;    // MONO_MAX_ITER of ReduceMonoCoeff (0 = fixed coefficient)
   R        gm1, inv_gm1, min_pres;
   int     *status;           // GB_INTERP_FAILED is OR-ed in where a parent still fails
};

// the conserved variables u of a coarse cell in place of its primitive ones, as Hydro_Con2Pri computes
// them for Interpolate_Iterate (src/Interpolation/Interpolate.cpp:250-262; CPU_Shared_FluUtility.cpp:209-296)
template <typename R>
GB_DEV void cell_primitive( const IntArgs<R> &a, R (&u)[5] )
{
   const R d = u[0], mx = u[1], my = u[2], mz = u[3];
   const R ird = rdiv( R(1), d );
   u[1] = rmul( mx, ird );  u[2] = rmul( my, ird );  u[3] = rmul( mz, ird );
   // Hydro_Con2Eint, EoS_DensEint2Pres_Gamma, Hydro_CheckMinPres
   const R eint = rsub( u[4], rdiv( rmul( R(0.5), radd( radd( rmul( mx, mx ), rmul( my, my ) ), rmul( mz, mz ) ) ), d ) );
   const R p = rmul( eint, a.gm1 );
   u[4] = ( p == p ) ? rmax( p, a.min_pres ) : p;
}

// the eight children f[fz][fy][fx] of the coarse cell c[0] of variable v; cx, cxy: strides along y and z
template <int SCH, typename R>
GB_DEV void children( const IntArgs<R> &a, const R *c, int cx, int cxy, int v, R coeff, R (&f)[2][2][2] )
{
   const bool mono = ( a.mono >> v ) & 1u, opp = a.opp != 0;
   if constexpr ( SCH == INT_MINMOD1D )
   {
      const R C = c[0];
      const R sx = minmod_slope( c[-1],   C, c[1],   opp );
      const R sy = minmod_slope( c[-cx],  C, c[cx],  opp );
      const R sz = minmod_slope( c[-cxy], C, c[cxy], opp );
#     pragma unroll
      for (int fz=0; fz<2; fz++)
#     pragma unroll
      for (int fy=0; fy<2; fy++)
#     pragma unroll
      for (int fx=0; fx<2; fx++)
      {
         R t = fz ? radd( C, sz ) : rsub( C, sz );
         t = fy ? radd( t, sy ) : rsub( t, sy );
         f[fz][fy][fx] = fx ? radd( t, sx ) : rsub( t, sx );
      }
   }
   else
   {
      constexpr int G = int_ghost( SCH ), W = 2*G + 1;
      R tx[W][W][2];         // x pass: [z][y][fine x]
#     pragma unroll
      for (int zz=0; zz<W; zz++)
#     pragma unroll
      for (int yy=0; yy<W; yy++)
      {
         R line[W];
         const R *q = c + ( zz - G )*cxy + ( yy - G )*cx;
#        pragma unroll
         for (int xx=0; xx<W; xx++) line[xx] = q[xx - G];
         op1d<SCH>( line, mono, coeff, opp, tx[zz][yy][0], tx[zz][yy][1] );
      }
      R ty[W][2][2];         // y pass: [z][fine y][fine x]
#     pragma unroll
      for (int zz=0; zz<W; zz++)
#     pragma unroll
      for (int fx=0; fx<2; fx++)
      {
         R line[W];
#        pragma unroll
         for (int yy=0; yy<W; yy++) line[yy] = tx[zz][yy][fx];
         op1d<SCH>( line, mono, coeff, opp, ty[zz][0][fx], ty[zz][1][fx] );
      }
#     pragma unroll
      for (int fy=0; fy<2; fy++)
#     pragma unroll
      for (int fx=0; fx<2; fx++)
      {
         R line[W];
#        pragma unroll
         for (int zz=0; zz<W; zz++) line[zz] = ty[zz][fy][fx];
         op1d<SCH>( line, mono, coeff, opp, f[0][fy][fx], f[1][fy][fx] );
      }
   }
}

// Interpolate(): every variable of every parent of the range, the fixed coefficient
template <int SCH, typename R>
__global__ void interp_kernel( const __grid_constant__ IntArgs<R> a )
{
   const int nx = a.crange[0], nxy = a.crange[0]*a.crange[1], ncell = nxy*a.crange[2];
   const size_t c3 = (size_t)a.csize[0]*a.csize[1]*a.csize[2], f3 = (size_t)a.fsize[0]*a.fsize[1]*a.fsize[2];
   for (long long t = blockIdx.x*(long long)blockDim.x + threadIdx.x; t < (long long)ncell*a.nbatch*a.ncomp;
        t += (long long)gridDim.x*blockDim.x)
   {
      const int c = (int)( t % ncell );
      const long long bv = t / ncell;
      const int v = (int)( bv % a.ncomp ), b = (int)( bv / a.ncomp );
      const int ii = c % nx, jj = ( c / nx ) % a.crange[1], kk = c / nxy;
      const int cx = a.csize[0], cxy = a.csize[0]*a.csize[1];
      const R *cb = a.cdata + ( (size_t)b*a.ncomp + v )*c3 + (size_t)( a.cstart[2] + kk )*cxy + ( a.cstart[1] + jj )*cx + a.cstart[0] + ii;
      R f[2][2][2];
      children<SCH>( a, cb, cx, cxy, v, a.mono_coeff, f );
      R *fb = a.fdata + ( (size_t)b*a.ncomp + v )*f3;
#     pragma unroll
      for (int fz=0; fz<2; fz++)
#     pragma unroll
      for (int fy=0; fy<2; fy++)
#     pragma unroll
      for (int fx=0; fx<2; fx++)
         fb[(size_t)( a.fstart[2] + 2*kk + fz )*a.fsize[0]*a.fsize[1] + ( a.fstart[1] + 2*jj + fy )*a.fsize[0] +
            ( a.fstart[0] + 2*ii + fx )] = f[fz][fy][fx];
   }
}

// Hydro_IsUnphysical of an interpolated child (src/Model_Hydro/CPU_Hydro/CPU_Shared_FluUtility.cpp:843-1010):
// conserved (with the internal-energy test) or primitive (then with the internal energy P/(gamma-1)
// of Interpolate_Iterate :399-430)
template <typename R>
GB_DEV bool child_fails( const IntArgs<R> &a, const R (&u)[5], bool prim )
{
   bool bad = false;
#  pragma unroll
   for (int v=0; v<5; v++)
   {
      bad |= ( u[v] != u[v] );
      if ( v >= 1 && v <= 3 ) bad |= ( u[v] < -Lim<R>::huge() || u[v] > Lim<R>::huge() );
      else if ( prim && v == 4 ) bad |= ( u[v] < R(0) || u[v] > Lim<R>::huge() );
      else                       bad |= ( u[v] <= R(0) || u[v] > Lim<R>::huge() );
   }
   if ( prim )
   {
      const R eint = rmul( u[4], a.inv_gm1 );
      bad |= ( eint < R(0) || eint > Lim<R>::huge() || eint != eint );
   }
   else
   {
      const R eint = rsub( u[4], rdiv( rmul( R(0.5), radd( radd( rmul( u[1], u[1] ), rmul( u[2], u[2] ) ), rmul( u[3], u[3] ) ) ), u[0] ) );
      bad |= ( eint < rmul( rmul( R(-3.0), u[4] ), Lim<R>::eps() ) || eint > Lim<R>::huge() || eint != eint );
   }
   return bad;
}

// Interpolate_Iterate for the five conserved hydro variables (INTERP_MASK: each parent on its own).
// One CTA takes a box of parents of one region, or several whole regions where they are small, with
// their coarse neighbourhoods in shared memory.  All parents of the CTA make the first attempt; those
// with an unphysical child are listed and make the next one together, in full warps, until none is
// left.  Before the second attempt the staged cells are turned into primitive variables in place, so
// that no stencil has to.  The children of the five variables stay in registers: with a run-time loop
// over the variables they went through local memory.  Bound by the issue of the 19 one-dimensional
// operators of a parent's variable, each of rounded multiplications and selects.
// cquad, FP32, us, against one thread per parent of the whole call that makes all its attempts from
// global memory: 342 regions of 12^3 cells 97 -> 54, with half of the parents iterating 233 -> 123; 4096:
// 1196 -> 565 and 2810 -> 1380; 8000 regions of 4^3 cells 25.4 -> 16.6 (with a CTA per region 251); one
// of 70^3 87.5 -> 80 (with a CTA per plane 172); a call of a few thousand parents, which is latency, 10.1 -> 10.2.
constexpr int INT_THREADS = 256;

// CTAs per SM: 342 regions of 12^3 cells, with the window assembly, us: FP32 1: 137, 2: 111, 3: 97, 4: 103
// (6 of 128 threads: 103); FP64 (229 regions) 1: 149, 2: 118, 3: 120, 4: 123
template <typename R> constexpr int int_ctas() { return sizeof(R) == 4 ? 3 : 2; }

// what a CTA takes: m whole regions, or (m = 1) one of nx x ny x nz boxes of n[] parents of a region
struct IntTile {
   int m, n[3], nbox[3];
   int b[3], cells;            // coarse cells staged per variable, along each axis and in all
   int list;                   // byte offset of the two lists of parents in shared memory
   int threads;
};

// one attempt of Interpolate_Iterate at the parent src[0] (variables vs apart), with its children stored at fo; false:
// a child came out unphysical and another attempt may follow.  LATER: an attempt after the first, in
// primitive variables if prim
template <int SCH, bool LATER, typename R>
GB_DEV bool int_attempt( const IntArgs<R> &a, const R *src, int sx, int sxy, int vs, R coeff, bool prim, bool more, R *fo, size_t fx,
                         size_t fxy, size_t f3 )
{
   R f[5][2][2][2];
#  pragma unroll
   for (int v=0; v<5; v++)
   {
      children<SCH>( a, src + v*vs, sx, sxy, v, coeff, f[v] );
      asm volatile( "" ::: "memory" );      // one variable's stencil live at a time
   }
   bool ok = true;
#  pragma unroll
   for (int q=0; q<8; q++)
   {
      R u[5];
#     pragma unroll
      for (int v=0; v<5; v++) u[v] = f[v][q >> 2][( q >> 1 ) & 1][q & 1];
      ok &= !child_fails( a, u, LATER && prim );
   }
   if ( !ok && more ) return false;
   if ( !ok ) atomicOr( a.status, GB_INTERP_FAILED );
   if ( LATER && prim )
   {
      // Hydro_Pri2Con: momenta rho*v, E = 1/2 |m|^2/rho + P/(gamma-1) (Hydro_ConEint2Etot)
#     pragma unroll
      for (int q=0; q<8; q++)
      {
         const int z = q >> 2, y = ( q >> 1 ) & 1, x = q & 1;
         const R d = f[0][z][y][x];
         const R mx = rmul( d, f[1][z][y][x] ), my = rmul( d, f[2][z][y][x] ), mz = rmul( d, f[3][z][y][x] );
         const R eint = rmul( f[4][z][y][x], a.inv_gm1 );
         f[1][z][y][x] = mx;  f[2][z][y][x] = my;  f[3][z][y][x] = mz;
         f[4][z][y][x] = radd( rdiv( rmul( R(0.5), radd( radd( rmul( mx, mx ), rmul( my, my ) ), rmul( mz, mz ) ) ), d ), eint );
      }
   }
   // (the two children along x, which share a sector, one after the other)
#  pragma unroll
   for (int v=0; v<5; v++)
#     pragma unroll
      for (int q=0; q<8; q++) fo[v*f3 + ( q >> 2 )*fxy + ( ( q >> 1 ) & 1 )*fx + ( q & 1 )] = f[v][q >> 2][( q >> 1 ) & 1][q & 1];
   return true;
}

template <int SCH, typename R>
__global__ void __launch_bounds__( INT_THREADS, int_ctas<R>() ) interp_iterate_kernel( const __grid_constant__ IntArgs<R> a,
                                                                                        const __grid_constant__ IntTile w )
{
   constexpr int G = int_ghost( SCH );
   extern __shared__ __align__(16) unsigned char int_smem[];
   __shared__ int s_nfail[2];
   R *s_c = (R*)int_smem;
   const int tid = threadIdx.x, nth = blockDim.x;
   // the region (the first of m) and the box of parents in it: its first parent and its extents
   int o[3] = { 0, 0, 0 }, p[3], bi = blockIdx.x;
   if ( w.nbox[0] > 1 ) { o[0] = ( bi % w.nbox[0] )*w.n[0];  bi /= w.nbox[0]; }
   if ( w.nbox[1] > 1 ) { o[1] = ( bi % w.nbox[1] )*w.n[1];  bi /= w.nbox[1]; }
   if ( w.nbox[2] > 1 ) { o[2] = ( bi % w.nbox[2] )*w.n[2];  bi /= w.nbox[2]; }
   const int b0 = bi*w.m, nreg = ( a.nbatch - b0 < w.m ) ? a.nbatch - b0 : w.m;
#  pragma unroll
   for (int d=0; d<3; d++) p[d] = ( a.crange[d] - o[d] < w.n[d] ) ? a.crange[d] - o[d] : w.n[d];
   const int sx = w.b[0], sxy = w.b[0]*w.b[1];
   const int cx = a.csize[0], cxy = a.csize[0]*a.csize[1];
   const size_t c3 = (size_t)cxy*a.csize[2];
   const int gx = a.cstart[0] + o[0] - G, gy = a.cstart[1] + o[1] - G, gz = a.cstart[2] + o[2] - G;
   if ( tid < 2 ) s_nfail[tid] = 0;
   if ( sx == cx && w.b[1] == a.csize[1] && ( w.m == 1 || w.b[2] == a.csize[2] ) )
   {
      // whole planes, one run per variable (one in all for several regions, which are whole); 16-byte loads
      // where every run starts on a 16-byte boundary
      constexpr int V = 16/sizeof(R);
      const R *src = a.cdata + (size_t)b0*5*c3 + (size_t)gz*cxy;
      const bool aligned = ( (uintptr_t)src & 15u ) == 0;
      if ( w.m == 1 )
      {
         const int len = ( p[2] + 2*G )*cxy, nv = ( aligned && c3 % V == 0 && w.cells % V == 0 ) ? len/V : 0;
         for (int e = tid; e < nv; e += nth)
#           pragma unroll
            for (int v=0; v<5; v++) ( (uint4*)( s_c + v*w.cells ) )[e] = ( (const uint4*)( src + v*c3 ) )[e];
         for (int e = nv*V + tid; e < len; e += nth)
#           pragma unroll
            for (int v=0; v<5; v++) s_c[v*w.cells + e] = src[v*c3 + e];
      }
      else
      {
         const int len = nreg*5*w.cells, nv = aligned ? len/V : 0;
#        pragma unroll 8
         for (int e = tid; e < nv; e += nth) ( (uint4*)s_c )[e] = ( (const uint4*)src )[e];
#        pragma unroll 8
         for (int e = nv*V + tid; e < len; e += nth) s_c[e] = src[e];
      }
   }
   else
   {
      const int bx = p[0] + 2*G, bxy = bx*( p[1] + 2*G ), bn = bxy*( p[2] + 2*G );
      for (int e = tid; e < nreg*bn; e += nth)
      {
         const int r = e / bn, c = e - r*bn, z = c / bxy, y = ( c - z*bxy ) / bx, x = c - z*bxy - y*bx;
         const R *src = a.cdata + (size_t)( b0 + r )*5*c3 + (size_t)( gz + z )*cxy + (size_t)( gy + y )*cx + gx + x;
         R *dst = s_c + r*5*w.cells + z*sxy + y*sx + x;
#        pragma unroll
         for (int v=0; v<5; v++) dst[v*w.cells] = src[v*c3];
      }
   }
   __syncthreads();

   const size_t fx = a.fsize[0], fxy = (size_t)a.fsize[0]*a.fsize[1], f3 = fxy*a.fsize[2];
   const int np = p[0]*p[1]*p[2], mono_iter = a.mono_max_iter, max_iter = a.int_prim ? mono_iter + 1 : mono_iter;
   unsigned short *list = (unsigned short*)( int_smem + w.list );        // [2][the CTA's parents]
   const int nlist = w.m*w.n[0]*w.n[1]*w.n[2];
   // Interpolate_Iterate stores from the origin of the fine region
   R *const f0 = a.fdata + (size_t)b0*5*f3 + (size_t)( 2*o[2] )*fxy + (size_t)( 2*o[1] )*fx + 2*o[0];
   // parent id of the CTA: its staged cell and its first child
   auto parent = [&]( int id, const R *&src, R *&fo )
   {
      unsigned c = id, kk, jj;
      src = s_c + G*( sxy + sx + 1 );
      fo = f0;
      if ( w.m > 1 )
      {
         const unsigned r = c / (unsigned)np;
         c -= r*np;
         src += r*5*w.cells;
         fo += r*5*f3;
      }
      jj = c / (unsigned)p[0];
      c -= jj*p[0];
      kk = jj / (unsigned)p[1];
      jj -= kk*p[1];
      src += kk*sxy + jj*sx + c;
      fo += 2*( kk*fxy + jj*fx + c );
   };
   int n = nreg*np;
   for (int id = tid; id < n; id += nth)
   {
      const R *src;
      R *fo;
      parent( id, src, fo );
      if ( !int_attempt<SCH,false>( a, src, sx, sxy, w.cells, a.mono_coeff, false, max_iter > 0, fo, fx, fxy, f3 ) )
         list[atomicAdd( &s_nfail[0], 1 )] = (unsigned short)id;
   }
   if ( max_iter == 0 ) return;
   R coeff = a.mono_coeff;
   for (int it=1; ; it++)
   {
      __syncthreads();
      n = s_nfail[( it + 1 ) & 1];
      if ( n == 0 ) return;
      if ( tid == 0 ) s_nfail[it & 1] = 0;
      if ( it == 1 && a.int_prim )
      {
         for (int e = tid; e < nreg*w.cells; e += nth)
         {
            R *q = s_c + ( e / w.cells )*5*w.cells + e % w.cells, u[5];
#           pragma unroll
            for (int v=0; v<5; v++) u[v] = q[v*w.cells];
            cell_primitive( a, u );
#           pragma unroll
            for (int v=0; v<5; v++) q[v*w.cells] = u[v];
         }
      }
      else coeff = rmax( rsub( coeff, rdiv( a.mono_coeff, (R)mono_iter ) ), R(0) );
      __syncthreads();
      const unsigned short *cur = list + ( ( it + 1 ) & 1 )*nlist;
      unsigned short *next = list + ( it & 1 )*nlist;
      for (int e = tid; e < n; e += nth)
      {
         const R *src;
         R *fo;
         parent( cur[e], src, fo );
         if ( !int_attempt<SCH,true>( a, src, sx, sxy, w.cells, coeff, a.int_prim != 0, it < max_iter, fo, fx, fxy, f3 ) )
            next[atomicAdd( &s_nfail[it & 1], 1 )] = cur[e];
      }
      if ( it == max_iter ) return;
   }
}

// The boxes of a call.  A round of 256 parents on an SM that holds a full set of CTAs takes one unit of
// time, alone on its SM `alone` units (measured for 12^3 regions: 8.3 and 11.7 us in FP32, 15 us both in
// FP64), the staging of 256 cells 0.06 (of a cell by one thread 0.03) and the launch of a CTA 0.05; the choice is the one for which the slowest SM, or the
// chain of rounds of the CTAs that follow each other in one place, takes least, and the largest box
// of those that tie.  At most 48 KB of shared memory.
template <typename R>
IntTile interp_tile( int scheme, const IntArgs<R> &a, int nsm )
{
   const int G = int_ghost( scheme );
   const double alone = ( sizeof(R) == 4 ) ? 1.4 : 1.0;
   constexpr int SMEM = 48*1024 - 64;
   const int nx = a.crange[0], ny = a.crange[1], nz = a.crange[2];
   const long long region = (long long)nx*ny*nz;
   IntTile best;
   best.m = 0;
   double best_cost = 0.0;
   // m regions, or a box of px x py x pz parents; whether it fits
   auto consider = [&]( int m, int px, int py, int pz )
   {
      const long long cells = (long long)( px + 2*G )*( py + 2*G )*( pz + 2*G ), parents = (long long)m*px*py*pz;
      const long long list = ( 5*m*cells*(long long)sizeof(R) + 15 )/16*16;
      if ( list + 4*parents > SMEM || parents > 65535 ) return false;
      IntTile t;
      t.m = m;
      t.n[0] = px;  t.n[1] = py;  t.n[2] = pz;
      for (int d=0; d<3; d++) { t.nbox[d] = ( a.crange[d] + t.n[d] - 1 )/t.n[d];  t.b[d] = t.n[d] + 2*G; }
      t.cells = (int)cells;
      t.list  = (int)list;
      const int rounds = (int)( ( parents + INT_THREADS - 1 )/INT_THREADS );
      const int warps = (int)( ( parents + 32*rounds - 1 )/( 32*rounds ) );
      t.threads = 32*warps;
      // CTAs that share an SM: by registers and by shared memory
      int share = int_ctas<R>()*( INT_THREADS/32 )/warps;
      const int fit = 227*1024/( t.list + 4*(int)parents + 1024 );
      if ( fit < share ) share = fit;
      const long long ctas = (long long)t.nbox[0]*t.nbox[1]*t.nbox[2]*( ( a.nbatch + m - 1 )/m );
      const long long per_sm = ( ctas + nsm - 1 )/nsm, waves = ( per_sm + share - 1 )/share;
      // threads beyond the parents stage the cells with fewer loads one after the other, where an SM has few CTAs
      int more = ( per_sm <= int_ctas<R>() ) ? INT_THREADS/32 : 0;
      if ( more > ( m*cells + 31 )/32 ) more = (int)( ( m*cells + 31 )/32 );
      if ( more > warps ) t.threads = 32*more;
      const double load = per_sm*( warps*rounds/8.0 + 0.06*m*cells/256 );
      const double chain = waves*( alone*rounds + 0.03*m*cells/t.threads );
      const double cost = ( ( load > chain ) ? load : chain ) + 0.05*per_sm;
      if ( best.m == 0 || cost < best_cost ) { best = t;  best_cost = cost; }
      return true;
   };
   // small regions: several, at most two rounds
   if ( region <= INT_THREADS )
      for (int m = ( a.nbatch < 2*INT_THREADS/(int)region ) ? a.nbatch : 2*INT_THREADS/(int)region; m > 1; m -= 1 + m/8) consider( m, nx, ny, nz );
   // whole planes, or boxes cut along y too where the planes are too large or too few for the SMs; along x
   // where not even one row fits, or only a box with less than a round of parents for a large region
   bool fits = false;
   for (int kx = 1; ; kx *= 2)
   {
      const int px = ( nx + kx - 1 )/kx;
      for (int ky = 1; ; ky *= 2)
      {
         const int py = ( ny + ky - 1 )/ky;
         int last = 0;
         for (int kz = 1; kz < 16 && kz <= nz; kz++)
         {
            const int pz = ( nz + kz - 1 )/kz;
            if ( pz != last ) fits |= consider( 1, px, py, pz );
            last = pz;
         }
         if ( last != 1 ) fits |= consider( 1, px, py, 1 );
         if ( py == 1 || ( fits && (long long)a.nbatch*ky*nz >= 2*nsm ) ) break;
      }
      if ( px == 1 || ( fits && ( px < 32 || best.threads >= INT_THREADS/2 || region*a.nbatch < (long long)nsm*INT_THREADS ) ) ) return best;
   }
}

template <int SCH, typename R>
cudaError_t iterate_launch( const IntArgs<R> &a, int nsm, cudaStream_t st )
{
   const IntTile t = interp_tile( SCH, a, nsm );
   const long long grid = (long long)t.nbox[0]*t.nbox[1]*t.nbox[2]*( ( a.nbatch + t.m - 1 )/t.m );
   if ( grid > 0x7fffffffLL ) return cudaErrorInvalidValue;
   const size_t smem = t.list + (size_t)4*t.m*t.n[0]*t.n[1]*t.n[2];
   interp_iterate_kernel<SCH,R><<< (unsigned)grid, t.threads, smem, st >>>( a, t );
   return cudaGetLastError();
}

template <typename R>
cudaError_t interp_launch( int scheme, bool iterate, const IntArgs<R> &a, cudaStream_t st )
{
   const long long ncell = (long long)a.crange[0]*a.crange[1]*a.crange[2];
   const long long items = ncell*a.nbatch*a.ncomp;
   constexpr int B = 128;
   long long g = ( items + B - 1 )/B;
   int dev = 0, nsm = 148;
   cudaGetDevice( &dev );
   cudaDeviceGetAttribute( &nsm, cudaDevAttrMultiProcessorCount, dev );
   if ( g > 32LL*nsm ) g = 32LL*nsm;
   if ( g < 1 ) return cudaSuccess;
#  define GB_INT_CASE( S ) \
   case S: if ( iterate ) return iterate_launch<S,R>( a, nsm, st ); \
           interp_kernel<S,R><<< (unsigned)g, B, 0, st >>>( a );  break;
   switch ( scheme )
   {
      GB_INT_CASE( INT_MINMOD3D )
      GB_INT_CASE( INT_MINMOD1D )
      GB_INT_CASE( INT_VANLEER )
      GB_INT_CASE( INT_CQUAD )
      GB_INT_CASE( INT_QUAD )
      GB_INT_CASE( INT_CQUAR )
      GB_INT_CASE( INT_QUAR )
      default: return cudaErrorInvalidValue;
   }
#  undef GB_INT_CASE
   return cudaGetLastError();
}

template <typename R>
int interp_run( const gb_interp_params *p, const void *cdata, void *fdata, int nbatch, cudaStream_t st )
{
   IntArgs<R> a;
   a.cdata = (const R*)cdata;  a.fdata = (R*)fdata;
   for (int d=0; d<3; d++)
   {
      a.csize[d] = p->csize[d];  a.cstart[d] = p->cstart[d];  a.crange[d] = p->crange[d];
      a.fsize[d] = p->fsize[d];  a.fstart[d] = p->fstart[d];
   }
   a.ncomp = p->ncomp;  a.nbatch = nbatch;
   a.mono = p->monotonic;  a.mono_coeff = (R)p->mono_coeff;  a.opp = p->opp_sign_0th_order;
   a.int_prim = p->int_prim;  a.mono_max_iter = p->mono_max_iter;
   // EoS_SetAuxArray_Gamma: constants formed in double, then cast
   a.gm1 = (R)( p->gamma - 1.0 );  a.inv_gm1 = (R)( 1.0/( p->gamma - 1.0 ) );  a.min_pres = (R)p->min_pres;
   a.status = p->status;
   // Interpolate() takes the iterative path only with IntPrim or ReduceMonoCoeff (Interpolate.cpp:152-156)
   const bool iterate = ( p->mode == GB_INTERP_ITERATE ) && ( p->int_prim || p->mono_max_iter > 0 );
   const cudaError_t e = interp_launch<R>( p->scheme, iterate, a, st );
   return ( e == cudaSuccess ) ? GB_OK : GB_E_CUDA;
}

// ---- window assembly of the ghost-zone fill ------------------------------------------------------
// Prepare_PatchData (src/Main/Prepare_PatchData.cpp) fills each side of a patch group's window from
// the patch groups of the same level where they exist and by interpolation from the coarser level
// where they do not (InterpolateGhostZone).  Here the side of a cell picks its source -- the patch
// group's own interior, the interior of the same-level patch group nbr[p][s], or the
// coarse-interpolated window cint[p] (gb_interpolate_device over the window).
//
// One CTA (of a few windows, several) fills the window of one variable of one patch group; the 27
// sources are resolved once into
// shared memory.  A thread writes four consecutive cells with 16-byte stores (VEC: a window is a
// whole number of them, since its width is even; an array that is not 16-byte aligned takes scalar
// stores).  NXT: the width, a constant for the usual ones, so that the index arithmetic divides by
// constants.  PAIR: cells are read two at a time (an even ghost width, so that a pair lies in one side,
// and sources aligned to a pair).
constexpr int ASM_THREADS = 256;

template <typename R, int NXT, bool VEC, bool PAIR>
__global__ void __launch_bounds__( ASM_THREADS ) assemble_windows_kernel( const R *fine, const int *nbr, const R *cint, R *win,
                                                                          int npg, int ncomp, int nxt_any )
{
   const int nxt = NXT ? NXT : nxt_any;
   const int g = ( nxt - PS2 )/2, n2 = nxt*nxt, n3 = nxt*n2;
   constexpr int PS3 = PS2*PS2*PS2;
   constexpr long long FROM_CINT = -1, NO_SOURCE = -2;
   __shared__ long long s_src[27];      // first element of the source interior, or one of the above
   for (long long pv = blockIdx.x; pv < (long long)npg*ncomp; pv += gridDim.x)
   {
      const int v = (int)( pv % ncomp ), p = (int)( pv / ncomp );
      __syncthreads();
      if ( threadIdx.x < 27 )
      {
         const int src = ( threadIdx.x == 13 ) ? p : nbr[(size_t)p*27 + threadIdx.x];
         // NO_SOURCE: not a patch group of the batch, or a coarse side without an interpolated window
         s_src[threadIdx.x] = ( src >= npg ) ? NO_SOURCE : ( src >= 0 ) ? ( (long long)src*ncomp + v )*PS3
                                                                         : ( cint != nullptr ) ? FROM_CINT : NO_SOURCE;
      }
      __syncthreads();
      const R *ci = cint + (size_t)pv*n3;
      R *wo = win + (size_t)pv*n3;
      for (int c0 = 4*( blockIdx.y*ASM_THREADS + threadIdx.x ); c0 < n3; c0 += 4*ASM_THREADS*gridDim.y)
      {
         constexpr int S = PAIR ? 2 : 1;
         R val[4];
#        pragma unroll
         for (int q=0; q<4; q += S)
         {
            const int c = c0 + q;
            const int k = c / n2, r = c - k*n2, j = r / nxt, i = r - j*nxt;
            const int x = i - g, y = j - g, z = k - g;
            const int dx = ( x < 0 ) ? -1 : ( x >= PS2 ), dy = ( y < 0 ) ? -1 : ( y >= PS2 ), dz = ( z < 0 ) ? -1 : ( z >= PS2 );
            const long long src = s_src[( dz + 1 )*9 + ( dy + 1 )*3 + ( dx + 1 )];
            const R *from = ( src >= 0 ) ? fine + src + ( ( z - PS2*dz )*PS2 + ( y - PS2*dy ) )*PS2 + ( x - PS2*dx )
                                         : ( src == FROM_CINT ) ? ci + c : nullptr;
            if constexpr ( PAIR )
            {
               typedef typename std::conditional<sizeof(R) == 4, float2, double2>::type R2;
               const R2 t = from ? *(const R2*)from : R2{ R(NAN), R(NAN) };
               val[q] = t.x;  val[q+1] = t.y;
            }
            else val[q] = from ? *from : R(NAN);
         }
         if constexpr ( !VEC )
         {
#           pragma unroll
            for (int q=0; q<4; q++) wo[c0 + q] = val[q];
         }
         else if constexpr ( sizeof(R) == 4 ) *(float4*)( wo + c0 ) = make_float4( val[0], val[1], val[2], val[3] );
         else { ( (double2*)( wo + c0 ) )[0] = make_double2( val[0], val[1] );  ( (double2*)( wo + c0 ) )[1] = make_double2( val[2], val[3] ); }
      }
   }
}

template <typename R>
int assemble_launch( const void *fine, const int *nbr, const void *cint, void *win, int npg, int ncomp, int nxt, cudaStream_t st )
{
   const long long items = (long long)npg*ncomp;
   // few windows: several CTAs each, about four per SM in all
   int dev = 0, nsm = 148;
   cudaGetDevice( &dev );
   cudaDeviceGetAttribute( &nsm, cudaDevAttrMultiProcessorCount, dev );
   const dim3 grid( (unsigned)( ( items < 0x7fffffffLL ) ? items : 0x7fffffffLL ),
                    (unsigned)( ( items >= 4*nsm ) ? 1 : ( 2*items <= nsm ) ? 8 : 4*nsm/items ) );
   const bool vec = ( (uintptr_t)win & 15u ) == 0;
   const bool pair = ( ( (uintptr_t)fine | (uintptr_t)cint ) & ( 2*sizeof(R) - 1 ) ) == 0;
#  define GB_ASM( N, V, P ) assemble_windows_kernel<R,N,V,P><<< grid, ASM_THREADS, 0, st >>>( (const R*)fine, nbr, (const R*)cint, (R*)win, npg, ncomp, nxt )
   if      ( !vec )              GB_ASM( 0, false, false );
   else if ( nxt == 20 && pair ) GB_ASM( 20, true, true );
   else if ( nxt == 24 && pair ) GB_ASM( 24, true, true );
   else if ( nxt == 22 )         GB_ASM( 22, true, false );
   else                          GB_ASM( 0, true, false );
#  undef GB_ASM
   return ( cudaGetLastError() == cudaSuccess ) ? GB_OK : GB_E_CUDA;
}

} // namespace
} // namespace gb

extern "C"
int gb_interpolate_device( const gb_interp_params *p, const void *cdata, void *fdata, int nbatch, void *stream )
{
   using namespace gb;
   if ( p == nullptr || nbatch < 0 ) return GB_E_INVALID;
   if ( nbatch == 0 ) return GB_OK;
   if ( cdata == nullptr || fdata == nullptr ) return GB_E_INVALID;
   if ( p->scheme < INT_MINMOD3D || p->scheme > INT_QUAR ) return ( p->scheme == 8 ) ? GB_E_UNSUPPORTED : GB_E_INVALID;
   if ( p->precision != GB_PREC_FP32 && p->precision != GB_PREC_FP64 ) return GB_E_INVALID;
   if ( p->ncomp < 1 || p->ncomp > 32 ) return GB_E_INVALID;
   if ( p->mode != GB_INTERP_PLAIN && p->mode != GB_INTERP_ITERATE ) return GB_E_INVALID;
   // the region the reference's Interpolate() accepts (Interpolate.cpp:104-117): CGhost coarse cells
   // around the range inside CData, the 2x finer range inside FData
   const int G = int_ghost( p->scheme );
   long long c3 = 1, f3 = 1;
   for (int d=0; d<3; d++)
   {
      if ( p->csize[d] < 1 || p->fsize[d] < 1 || p->crange[d] < 1 ) return GB_E_INVALID;
      if ( p->cstart[d] < G || p->cstart[d] + p->crange[d] > p->csize[d] - G ) return GB_E_INVALID;
      if ( p->fstart[d] < 0 || p->fstart[d] + 2*p->crange[d] > p->fsize[d] ) return GB_E_INVALID;
      c3 *= p->csize[d];  f3 *= p->fsize[d];
   }
   if ( c3*p->ncomp*nbatch > 0x7fffffffLL*8 || f3*p->ncomp*nbatch > 0x7fffffffLL*8 ) return GB_E_INVALID;
   if ( p->mode == GB_INTERP_ITERATE )
   {
      // Interpolate_Iterate: all five conserved hydro variables, the fine region from the origin
      // (Interpolate.cpp:218-220), a positive gamma - 1, the failure flag; the reference refuses to
      // reduce the coefficient of MinMod-3D/1D and vanLeer (:273-276)
      if ( p->ncomp != 5 || p->status == nullptr || !( p->gamma > 1.0 ) || p->mono_max_iter < 0 ) return GB_E_INVALID;
      if ( p->fstart[0] || p->fstart[1] || p->fstart[2] ) return GB_E_INVALID;
      if ( p->mono_max_iter > 0 && ( p->scheme == INT_MINMOD3D || p->scheme == INT_MINMOD1D || p->scheme == INT_VANLEER ) )
         return GB_E_INVALID;
   }
   if ( p->precision == GB_PREC_FP64 ) return interp_run<double>( p, cdata, fdata, nbatch, (cudaStream_t)stream );
   return interp_run<float>( p, cdata, fdata, nbatch, (cudaStream_t)stream );
}

extern "C"
int gb_assemble_windows_device( const void *fine, const int *nbr, const void *cint, void *windows, int npg, int ncomp,
                                int nxt, int precision, void *stream )
{
   using namespace gb;
   if ( npg < 0 || ncomp < 1 || nxt < PS2 + 2 || nxt > PS2 + 2*PS2 || ( nxt - PS2 ) % 2 != 0 ) return GB_E_INVALID;
   if ( precision != GB_PREC_FP32 && precision != GB_PREC_FP64 ) return GB_E_INVALID;
   if ( npg == 0 ) return GB_OK;
   if ( fine == nullptr || nbr == nullptr || windows == nullptr ) return GB_E_INVALID;
   cudaStream_t st = (cudaStream_t)stream;
   return ( precision == GB_PREC_FP64 ) ? assemble_launch<double>( fine, nbr, cint, windows, npg, ncomp, nxt, st )
                                        : assemble_launch<float> ( fine, nbr, cint, windows, npg, ncomp, nxt, st );
}
