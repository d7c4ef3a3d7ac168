// Elementwise P1 operator for -div(k grad u) with optional icosahedral-shell blending (sm_100a).
//
// Reference: P1ElementwiseOperator with the HyTeG form p1_div_k_grad_blending_q3
// (src/hyteg/elementwiseoperators/P1ElementwiseOperator.cpp, src/hyteg/forms/form_hyteg_generated/p1/
// p1_div_k_grad_blending_q3.cpp): every micro-cell gets its 4x4 element matrix from a 5-point
// degree-3 quadrature (Yu's rule: centroid weight -2/15, four points with barycentric weights
// (1/2, 1/6, 1/6, 1/6) and weight 3/40), the coefficient is evaluated at the blended (physical)
// quadrature point and the blending Jacobian enters the gradients and the volume factor.
//
// GPU scheme: the micro-cells of a macro-cell are grouped by the parity of their anchor index; two
// anchors of the same parity differ by at least 2 in some coordinate, so the micro-cells of one
// parity class never share a vertex and a thread can add its element contributions without atomics.
// Eight passes (one per parity) accumulate A x into a scratch array laid out like the function; a
// combine kernel then applies the same epilogues as the constant-stencil path (apply, residual,
// Jacobi, Chebyshev steps) with a per-DoF inverse diagonal, summing the cell copies of face, edge
// and vertex DoFs into their owners (the additive communication of the reference).  Deterministic:
// the order of every sum is fixed.  The path is FP64-compute-bound.
#include "hyb_internal.hpp"
#include "p2_stored.cuh"

#include <cmath>
#include <stdexcept>

namespace hyb {

// ---------------------------------------------------------------------------------------------
// host: cell geometry and IcosahedralShellMap classification
// ---------------------------------------------------------------------------------------------
static void cross3( const double* a, const double* b, double* c )
{
   c[0] = a[1] * b[2] - a[2] * b[1];
   c[1] = a[2] * b[0] - a[0] * b[2];
   c[2] = a[0] * b[1] - a[1] * b[0];
}

// IcosahedralShellMap::classifyVertices (geometry/IcosahedralShellMap.hpp:606-705): the two vertices
// on a radial ray become ref/ray (ref is the single outer vertex of an outward tet, the single inner
// vertex of an inward tet); skew tets borrow the classification of a non-skew tet of the same prism.
static void classify_shell( const Topology& t, int c, CellGeom& g, int depth = 0 )
{
   if ( depth > 4 ) throw std::runtime_error( "shell blending: cannot classify macro-cell" );
   double P[4][3], rad[4];
   for ( int k = 0; k < 4; ++k )
   {
      for ( int d = 0; d < 3; ++d ) P[k][d] = t.vx[t.cv[c][k]][d];
      rad[k] = std::sqrt( P[k][0] * P[k][0] + P[k][1] * P[k][1] + P[k][2] * P[k][2] );
   }
   double inner = rad[0], outer = rad[0];
   for ( int k = 1; k < 4; ++k ) inner = std::min( inner, rad[k] ), outer = std::max( outer, rad[k] );
   const double eps     = ( outer - inner ) * 0.001;
   int          n_outer = 0;
   for ( int k = 0; k < 4; ++k ) n_outer += ( outer - rad[k] ) < eps ? 1 : 0;
   int iref = -1, iray = -1;
   for ( int k = 0; k < 4 && iref < 0; ++k )
      for ( int j = k + 1; j < 4 && iref < 0; ++j )
      {
         double cr[3];
         cross3( P[k], P[j], cr );
         const double s = rad[k] * rad[j];
         if ( std::fabs( cr[0] ) / s <= 1e-14 && std::fabs( cr[1] ) / s <= 1e-14 && std::fabs( cr[2] ) / s <= 1e-14 ) iref = k, iray = j;
      }
   if ( iref < 0 ) throw std::runtime_error( "shell blending: no radial vertex pair in a macro-cell (not a shell mesh?)" );
   if ( n_outer == 2 )
   {
      const int vref = t.cv[c][iref], vray = t.cv[c][iray];
      for ( int f : t.cf[c] )
      {
         const auto& fv     = t.fv[f];
         const bool  hasRef = fv[0] == vref || fv[1] == vref || fv[2] == vref;
         const bool  hasRay = fv[0] == vray || fv[1] == vray || fv[2] == vray;
         if ( !( hasRef && hasRay ) )
            for ( int cc : t.f_cells[f] )
               if ( cc != c ) return classify_shell( t, cc, g, depth + 1 );
      }
      throw std::runtime_error( "shell blending: no non-skew neighbour" );
   }
   int rest[2], nr = 0;
   for ( int k = 0; k < 4; ++k )
      if ( k != iref && k != iray ) rest[nr++] = k;
   const int ithr = rest[1], ifor = rest[0];
   if ( ( n_outer == 1 && rad[iref] < rad[iray] ) || ( n_outer == 3 && rad[iref] > rad[iray] ) ) std::swap( iref, iray );
   double a[3], b[3];
   for ( int d = 0; d < 3; ++d )
   {
      g.ray[d] = P[iray][d];
      a[d]     = P[ithr][d] - P[iray][d];
      b[d]     = P[ifor][d] - P[iray][d];
   }
   cross3( a, b, g.bxc );
   g.volT    = ( P[iref][0] - P[iray][0] ) * g.bxc[0] + ( P[iref][1] - P[iray][1] ) * g.bxc[1] + ( P[iref][2] - P[iray][2] ) * g.bxc[2];
   g.rad_ray = rad[iray];
   g.rad_ref = rad[iref];
}

void cell_geometry( const Topology& t, int c, int blending, CellGeom& g )
{
   g = CellGeom{};
   for ( int k = 0; k < 4; ++k )
      for ( int d = 0; d < 3; ++d ) g.P[k][d] = t.vx[t.cv[c][k]][d];
   g.blend = blending;
   if ( blending == 1 ) classify_shell( t, c, g );
}

void build_elementwise_operator( Operator* A )
{
   const Topology& t = A->mesh->topo;
   A->geom.assign( t.nC, CellGeom{} );
   for ( int c = 0; c < t.nC; ++c ) cell_geometry( t, c, A->blending, A->geom[c] );
}

// ---------------------------------------------------------------------------------------------
// device: blending, coefficient and element matrix
// ---------------------------------------------------------------------------------------------
__constant__ double c_yu5_pts[5][3] = { { 0.25, 0.25, 0.25 },
                                        { 1.0 / 6.0, 1.0 / 6.0, 1.0 / 6.0 },
                                        { 0.5, 1.0 / 6.0, 1.0 / 6.0 },
                                        { 1.0 / 6.0, 0.5, 1.0 / 6.0 },
                                        { 1.0 / 6.0, 1.0 / 6.0, 0.5 } };
__constant__ double c_yu5_w[5]      = { -2.0 / 15.0, 3.0 / 40.0, 3.0 / 40.0, 3.0 / 40.0, 3.0 / 40.0 };

// sin and cos of 2 pi f (x + p) go through sinpi / cospi, which need no reduction by an irrational
// period: fewer instructions than sin and cos, and no error from the rounded 2 pi f
__device__ __forceinline__ double sin_pi( double v ) { return sinpi( v ); }
__device__ __forceinline__ float  sin_pi( float v ) { return sinpif( v ); }
__device__ __forceinline__ double cos_pi( double v ) { return cospi( v ); }
__device__ __forceinline__ float  cos_pi( float v ) { return cospif( v ); }

// radius: |P| where the caller has it, or a negative value
template < typename A >
__device__ __forceinline__ A coeff_eval( const Coefficient& k, const A* P, A radius = A( -1 ) )
{
   if ( k.kind == 0 ) return A( k.value );
   if ( k.kind == 2 )  // radial profile exp(amp (value - |x|) / freq)
   {
      if ( radius < A( 0 ) ) radius = sqrt( P[0] * P[0] + P[1] * P[1] + P[2] * P[2] );
      return exp( A( k.amp / k.freq ) * ( A( k.value ) - radius ) );
   }
   const A tf = A( 2.0 * k.freq );
   return exp( A( k.amp ) * sin_pi( tf * ( P[0] + A( k.phase[0] ) ) ) * cos_pi( tf * ( P[1] + A( k.phase[1] ) ) ) *
               sin_pi( tf * ( P[2] + A( k.phase[2] ) ) ) );
}

// IcosahedralShellMap: F(x) = x r(x)/|x|, r(x) = r_ray + lambda(x) (r_ref - r_ray) with lambda the
// barycentric weight of the ref vertex; DF = s I + x (grad s)^T with s = r/|x|.
template < typename A >
__device__ __forceinline__ void shell_map( const CellGeom& g, const A* X, A* F, A DF[3][3] )
{
   const A dx = X[0] - A( g.ray[0] ), dy = X[1] - A( g.ray[1] ), dz = X[2] - A( g.ray[2] );
   const A lam_s = ( dx * A( g.bxc[0] ) + dy * A( g.bxc[1] ) + dz * A( g.bxc[2] ) ) / A( g.volT );
   const A sgn   = lam_s < A( 0 ) ? A( -1 ) : A( 1 );
   const A dr    = A( g.rad_ref ) - A( g.rad_ray );
   const A R     = A( g.rad_ray ) + fabs( lam_s ) * dr;
   const A r2    = X[0] * X[0] + X[1] * X[1] + X[2] * X[2];
   const A r     = sqrt( r2 );
   const A s     = R / r;
   A       gs[3];
   for ( int j = 0; j < 3; ++j ) gs[j] = ( dr * sgn * A( g.bxc[j] ) / A( g.volT ) ) / r - R * X[j] / ( r2 * r );
   for ( int i = 0; i < 3; ++i )
   {
      F[i] = X[i] * s;
      for ( int j = 0; j < 3; ++j ) DF[i][j] = ( i == j ? s : A( 0 ) ) + X[i] * gs[j];
   }
}

// P1 PSPG stabilisation element matrix of an affine micro-cell (form p1_tet_pspg_tet.h, whose inverted
// diagonal P1PSPGInvDiagOperator scales the Uzawa pressure update): -(|T|^(2/3) / 12) |T| grad l_i .
// grad l_j, the l_i barycentric coordinates and |T| the volume.  Exact (constant integrand).
template < typename A >
__device__ __forceinline__ void p1_pspg_element( const A X[4][3], A K[4][4] )
{
   A J[3][3];
   for ( int r = 0; r < 3; ++r )
      for ( int c = 0; c < 3; ++c ) J[r][c] = X[c + 1][r] - X[0][r];
   const A c00 = J[1][1] * J[2][2] - J[1][2] * J[2][1], c01 = J[1][2] * J[2][0] - J[1][0] * J[2][2],
           c02 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
   const A det = J[0][0] * c00 + J[0][1] * c01 + J[0][2] * c02;
   // rows of J^-1 are the gradients of l_1, l_2, l_3
   A G[4][3];
   G[1][0] = c00 / det, G[1][1] = ( J[0][2] * J[2][1] - J[0][1] * J[2][2] ) / det, G[1][2] = ( J[0][1] * J[1][2] - J[0][2] * J[1][1] ) / det;
   G[2][0] = c01 / det, G[2][1] = ( J[0][0] * J[2][2] - J[0][2] * J[2][0] ) / det, G[2][2] = ( J[0][2] * J[1][0] - J[0][0] * J[1][2] ) / det;
   G[3][0] = c02 / det, G[3][1] = ( J[0][1] * J[2][0] - J[0][0] * J[2][1] ) / det, G[3][2] = ( J[0][0] * J[1][1] - J[0][1] * J[1][0] ) / det;
   for ( int d = 0; d < 3; ++d ) G[0][d] = -( G[1][d] + G[2][d] + G[3][d] );
   const A vol = fabs( det ) / A( 6 );
   const A f   = -( pow( vol, A( 2.0 / 3.0 ) ) / A( 12 ) ) * vol;
   for ( int i = 0; i < 4; ++i )
      for ( int j = 0; j < 4; ++j ) K[i][j] = f * ( G[i][0] * G[j][0] + G[i][1] * G[j][1] + G[i][2] * G[j][2] );
}

// Minus the lumped P1 mass matrix weighted by 1/k, diag_i = -int l_i / k over the (blended) micro-cell
// (Yu's 5-point degree-3 rule): with k the viscosity, the scaling of the pressure update that follows
// the viscosity-weighted pressure mass matrix, the usual approximation of the Schur complement
// B A^-1 B^T for variable viscosity (negative like the PSPG diagonal, so the Uzawa update keeps its sign).
template < typename A >
__device__ __forceinline__ void p1_lumped_mass_inv_k_element( const CellGeom& g, const Coefficient& kc, const A X[4][3], A K[4][4] )
{
   A J[3][3];
   for ( int r = 0; r < 3; ++r )
      for ( int c = 0; c < 3; ++c ) J[r][c] = X[c + 1][r] - X[0][r];
   for ( int i = 0; i < 4; ++i )
      for ( int j = 0; j < 4; ++j ) K[i][j] = A( 0 );
#pragma unroll 1
   for ( int q = 0; q < 5; ++q )
   {
      const A xi[3] = { A( c_yu5_pts[q][0] ), A( c_yu5_pts[q][1] ), A( c_yu5_pts[q][2] ) };
      A       Xq[3];
      for ( int r = 0; r < 3; ++r ) Xq[r] = X[0][r] + J[r][0] * xi[0] + J[r][1] * xi[1] + J[r][2] * xi[2];
      A M[3][3], Fq[3];
      if ( g.blend == 1 )
      {
         A DF[3][3];
         shell_map( g, Xq, Fq, DF );
         for ( int r = 0; r < 3; ++r )
            for ( int c = 0; c < 3; ++c ) M[r][c] = DF[r][0] * J[0][c] + DF[r][1] * J[1][c] + DF[r][2] * J[2][c];
      }
      else
         for ( int r = 0; r < 3; ++r )
         {
            Fq[r] = Xq[r];
            for ( int c = 0; c < 3; ++c ) M[r][c] = J[r][c];
         }
      const A det = M[0][0] * ( M[1][1] * M[2][2] - M[1][2] * M[2][1] ) - M[0][1] * ( M[1][0] * M[2][2] - M[1][2] * M[2][0] ) +
                    M[0][2] * ( M[1][0] * M[2][1] - M[1][1] * M[2][0] );
      const A f     = A( c_yu5_w[q] ) * fabs( det ) / coeff_eval( kc, Fq );
      const A lam[4] = { A( 1 ) - xi[0] - xi[1] - xi[2], xi[0], xi[1], xi[2] };
      for ( int i = 0; i < 4; ++i ) K[i][i] -= f * lam[i];
   }
}

template < typename A >
__device__ __forceinline__ void p1_divkgrad_element( const CellGeom& g, const Coefficient& kc, const A X[4][3], A K[4][4] )
{
   A J[3][3];
   for ( int r = 0; r < 3; ++r )
      for ( int c = 0; c < 3; ++c ) J[r][c] = X[c + 1][r] - X[0][r];
   for ( int i = 0; i < 4; ++i )
      for ( int j = 0; j < 4; ++j ) K[i][j] = A( 0 );
#pragma unroll 1
   for ( int q = 0; q < 5; ++q )
   {
      A Xq[3];
      for ( int r = 0; r < 3; ++r )
         Xq[r] = X[0][r] + J[r][0] * A( c_yu5_pts[q][0] ) + J[r][1] * A( c_yu5_pts[q][1] ) + J[r][2] * A( c_yu5_pts[q][2] );
      A M[3][3], Fq[3];
      if ( g.blend == 1 )
      {
         A DF[3][3];
         shell_map( g, Xq, Fq, DF );
         for ( int r = 0; r < 3; ++r )
            for ( int c = 0; c < 3; ++c ) M[r][c] = DF[r][0] * J[0][c] + DF[r][1] * J[1][c] + DF[r][2] * J[2][c];
      }
      else
      {
         for ( int r = 0; r < 3; ++r )
         {
            Fq[r] = Xq[r];
            for ( int c = 0; c < 3; ++c ) M[r][c] = J[r][c];
         }
      }
      // inverse of M: rows of M^-1 are the reference gradients mapped to physical space
      const A c00 = M[1][1] * M[2][2] - M[1][2] * M[2][1];
      const A c01 = M[1][2] * M[2][0] - M[1][0] * M[2][2];
      const A c02 = M[1][0] * M[2][1] - M[1][1] * M[2][0];
      const A det = M[0][0] * c00 + M[0][1] * c01 + M[0][2] * c02;
      const A id  = A( 1 ) / det;
      A       Mi[3][3];
      Mi[0][0] = c00 * id;
      Mi[1][0] = c01 * id;
      Mi[2][0] = c02 * id;
      Mi[0][1] = ( M[0][2] * M[2][1] - M[0][1] * M[2][2] ) * id;
      Mi[1][1] = ( M[0][0] * M[2][2] - M[0][2] * M[2][0] ) * id;
      Mi[2][1] = ( M[0][1] * M[2][0] - M[0][0] * M[2][1] ) * id;
      Mi[0][2] = ( M[0][1] * M[1][2] - M[0][2] * M[1][1] ) * id;
      Mi[1][2] = ( M[0][2] * M[1][0] - M[0][0] * M[1][2] ) * id;
      Mi[2][2] = ( M[0][0] * M[1][1] - M[0][1] * M[1][0] ) * id;
      // gradient of phi_i (i = 1..3) is row i-1 of Mi; phi_0 is minus their sum
      A G[4][3];
      for ( int d = 0; d < 3; ++d )
      {
         G[1][d] = Mi[0][d];
         G[2][d] = Mi[1][d];
         G[3][d] = Mi[2][d];
         G[0][d] = -( G[1][d] + G[2][d] + G[3][d] );
      }
      const A f = A( c_yu5_w[q] ) * coeff_eval( kc, Fq ) * fabs( det );
      for ( int i = 0; i < 4; ++i )
         for ( int j = i; j < 4; ++j ) K[i][j] += f * ( G[i][0] * G[j][0] + G[i][1] * G[j][1] + G[i][2] * G[j][2] );
   }
   for ( int i = 0; i < 4; ++i )
      for ( int j = 0; j < i; ++j ) K[i][j] = K[j][i];
}

}  // namespace hyb

namespace hyb {

// micro-cell types: vertex offsets and anchor range shift (CellDoFIndexing.hpp:155-198)
__constant__ int c_mc_off[6][4][3] = {
    { { 0, 0, 0 }, { 1, 0, 0 }, { 0, 1, 0 }, { 0, 0, 1 } }, { { 1, 0, 0 }, { 1, 1, 0 }, { 0, 1, 0 }, { 1, 0, 1 } },
    { { 1, 0, 0 }, { 0, 1, 0 }, { 1, 0, 1 }, { 0, 0, 1 } }, { { 1, 1, 0 }, { 1, 1, 1 }, { 0, 1, 1 }, { 1, 0, 1 } },
    { { 1, 0, 1 }, { 0, 1, 1 }, { 0, 0, 1 }, { 0, 1, 0 } }, { { 0, 1, 0 }, { 1, 1, 0 }, { 1, 0, 1 }, { 0, 1, 1 } } };
__constant__ int c_mc_shift[6] = { 0, 1, 1, 2, 1, 1 };
// stencil direction (index into kVarDirs) from vertex i to vertex j of micro-cell type ty
__constant__ __align__( 16 ) int8_t c_mc_dir[6][4][4];
// the 15 stencil directions in the order of the constant-stencil weights
static const int kVarDirs[15][3] = { { 0, 0, 0 },  { -1, 0, 0 }, { 1, 0, 0 },  { 0, -1, 0 }, { 0, 1, 0 },
                                     { 0, 0, -1 }, { 0, 0, 1 },  { -1, 1, 0 }, { 1, -1, 0 }, { -1, 0, 1 },
                                     { 1, 0, -1 }, { 0, -1, 1 }, { 0, 1, -1 }, { 1, -1, 1 }, { -1, 1, -1 } };

__device__ __forceinline__ double ld_any( const double* p ) { return *p; }
__device__ __forceinline__ float  ld_any( const float* p ) { return *p; }
__device__ __forceinline__ float  ld_any( const __half* p ) { return __half2float( *p ); }
__device__ __forceinline__ void   st_any( double* p, double v ) { *p = v; }
__device__ __forceinline__ void   st_any( float* p, float v ) { *p = v; }
__device__ __forceinline__ void   st_any( __half* p, float v ) { *p = __float2half_rn( v ); }

// One parity pass: a thread per micro-cell anchor of the class (blocks of one macro-cell) and its micro-cells in
// order.  FP64: 168 registers, so that three blocks of 128 fit an SM; at 170 two did (shell of 1920 cells, level 4,
// exp/sin coefficient: 2.45 ms at 155 registers with sin and cos, 3.15 with sinpi at 170, 2.26 so).  FP32: six blocks
// (1.09 ms there; without the bound the compiler takes more registers: 1.21).
// MODE 0: y += K x with K computed on the fly; 1: diagonal of K; 4: add K into the assembled stencils of
// the cell-array slots of its vertices (kst = stencils, kstride = level size).
template < typename T, typename A, int MODE >
__global__ void __launch_bounds__( 128, sizeof( A ) == 8 ? 3 : 6 ) k_elem_pass( int n, int nanch, const int* __restrict__ anch, const int64_t* __restrict__ cell_off,
                                                       const CellGeom* __restrict__ geom, Coefficient kc,
                                                       const T* __restrict__ src, A* __restrict__ acc, A* __restrict__ kst,
                                                       int64_t kstride, int64_t level_size, int* err )
{
   const int t = blockIdx.x * blockDim.x + threadIdx.x;  // one micro-cell anchor per thread
   const int c = blockIdx.y;
   if ( t >= nanch ) return;
   const int      a = anch[t];
   const int      x = a & 1023, y = ( a >> 10 ) & 1023, z = a >> 20;
   const CellGeom g  = geom[c];
   const int64_t  base = cell_off[c];
   const A        inv_n = A( 1.0 / double( n ) );
   A              st[3][3];  // computational steps per index direction (coordinateFromIndex)
   for ( int k = 0; k < 3; ++k )
      for ( int d = 0; d < 3; ++d ) st[k][d] = ( A( g.P[k + 1][d] ) - A( g.P[0][d] ) ) * inv_n;
      for ( int ty = 0; ty < 6; ++ty )
      {
         if ( x + y + z > n - 1 - c_mc_shift[ty] ) continue;
         int64_t idx[4];
         A       X[4][3];
         for ( int m = 0; m < 4; ++m )
         {
            const int vx = x + c_mc_off[ty][m][0], vy = y + c_mc_off[ty][m][1], vz = z + c_mc_off[ty][m][2];
            idx[m]       = base + cidx( n, vx, vy, vz );
            for ( int d = 0; d < 3; ++d ) X[m][d] = A( g.P[0][d] ) + st[0][d] * A( vx ) + st[1][d] * A( vy ) + st[2][d] * A( vz );
         }
         A K[4][4];
         // self-check: every node inside the level's vector; a violation is recorded (error word 2) and
         // the micro-cell skipped
         {
            bool bad = false;
            for ( int m = 0; m < 4; ++m ) bad |= idx[m] < 0 || idx[m] >= level_size;
            if ( bad )
            {
               atomicExch( err, 2 );
               continue;
            }
         }
         if ( kc.kind == kCoeffPSPG ) p1_pspg_element( X, K );
         else if ( kc.element == kElemLumpedMassInvK ) p1_lumped_mass_inv_k_element( g, kc, X, K );
         else p1_divkgrad_element( g, kc, X, K );
         if constexpr ( MODE == 0 )
         {
            A xl[4];
            for ( int m = 0; m < 4; ++m ) xl[m] = A( ld_any( src + idx[m] ) );
            for ( int i = 0; i < 4; ++i ) acc[idx[i]] += K[i][0] * xl[0] + K[i][1] * xl[1] + K[i][2] * xl[2] + K[i][3] * xl[3];
         }
         else if constexpr ( MODE == 1 )
            for ( int i = 0; i < 4; ++i ) acc[idx[i]] += K[i][i];
         else if constexpr ( MODE == 4 )
            for ( int i = 0; i < 4; ++i )
               for ( int j = 0; j < 4; ++j )
               {
                  const int d = c_mc_dir[ty][i][j];  // opposite directions: the one with the even number is kept
                  if ( !( d & 1 ) ) kst[int64_t( d / 2 ) * kstride + idx[i]] += K[i][j];
               }
      }
}

// ---------------------------------------------------------------------------------------------
// P2 elementwise operators (P2ElementwiseOperator::apply / computeDiagonalOperatorValues,
// elementwiseoperators/P2ElementwiseOperator.cpp:109-318,418-567) with p2_div_k_grad_blending_q4.
// A P2 function on level L is stored on the node set of level L+1: the level-L micro-cell with
// vertices v0..v3 has its ten nodes at 2 v_i (vertices) and v_i + v_j (edge midpoints, edge order
// (2,3), (1,3), (1,2), (0,3), (0,2), (0,1)) in storage coordinates.  Element integrals use the
// degree-4, 11-point Xiao-Gimbutas rule on the tetrahedron, the rule the reference's form is
// generated with; its weights are derived here from exactness for all polynomials of degree <= 4.
// ---------------------------------------------------------------------------------------------
__constant__ double c_xg4_pts[11][3];
__constant__ double c_xg4_bary[11][4];
__constant__ double c_xg4_w[11];
__constant__ double c_xg4_mass[11][10];  // w lambda_i lambda_j, i <= j
__constant__ __align__( 16 ) int8_t c_p2_from[60];     // micro-cell nodes 10 ty + i, grouped by the window node they are
__constant__ __align__( 16 ) int8_t c_p2_from0[28];    // window node l: entries c_p2_from0[l] .. c_p2_from0[l + 1] - 1
__constant__ __align__( 16 ) int8_t c_p2_loc[6][10];  // node of micro-cell type ty in its anchor's 3x3x3 nodes: a + 3 b + 9 c
__constant__ double c_p2_rgrad[11][10][3];  // reference gradients of the ten basis functions per point
__constant__ double c_p2_phi[11][10];       // values of the ten basis functions per point
__constant__ int    c_p2_edge[6][2] = { { 2, 3 }, { 1, 3 }, { 1, 2 }, { 0, 3 }, { 0, 2 }, { 0, 1 } };
__constant__ __align__( 16 ) int8_t c_p2_node0[27];   // node of micro-cell type 0 at a window node, or -1
__constant__ __align__( 16 ) int8_t c_p2s_ent[600];  // entry of node j in node i's class stencil: (10 ty + i) 10 + j

// barycentric coordinates (l0, l1, l2, l3) of the rule's points (kept identical to the reference's
// generated form: the element integrals must agree); reference coordinates are (l1, l2, l3)
static const double kXG4Bary[11][4] = {
    { 0.17469405869723054, 0.04049050672759043, 0.01356070187980288, 0.7712547326953761 },
    { 0.08140491840285922, 0.752508507009655, 0.06809937093820666, 0.09798720364927911 },
    { 0.3044484024344971, 0.2402766649280726, 0.126801725915392, 0.3284732067220384 },
    { 0.7412288820936226, 0.0672232948933834, 0.03518392977359872, 0.1563638932393953 },
    { 0.053341239535745266, 0.419266313879513, 0.04778143555908666, 0.4796110110256551 },
    { 0.4329534904813558, 0.4507658760912768, 0.05945661629943383, 0.05682401712793367 },
    { 0.5380072039161857, 0.1294113737889104, 0.3301904148374645, 0.002391007457439365 },
    { 0.008991260093335729, 0.1215419913339278, 0.3064939884296903, 0.5629727601430461 },
    { 0.10660417256199362, 0.09720464458758327, 0.68439041545304, 0.1118007673973831 },
    { 0.3292329597426468, 0.02956949520647961, 0.3179035602133946, 0.323293984837479 },
    { 0.10384411641099309, 0.4327102390477686, 0.3538232392092971, 0.1096224053319412 } };

// weights w solving sum_q w_q xi_q^a = a1! a2! a3! / (|a|+3)! for all |a| <= 4 in the least-squares
// sense (Householder QR of the 35 x 11 moment matrix; exact for a degree-4 rule)
static void xg4_weights( double w[11] )
{
   const int           m = 35, n = 11;
   std::vector< double > A( m * n ), b( m );
   auto fact = []( int k ) {
      double f = 1;
      for ( int i = 2; i <= k; ++i ) f *= i;
      return f;
   };
   int row = 0;
   for ( int a = 0; a <= 4; ++a )
      for ( int bb = 0; bb <= 4 - a; ++bb )
         for ( int c = 0; c <= 4 - a - bb; ++c, ++row )
         {
            for ( int q = 0; q < n; ++q )
               A[row * n + q] = std::pow( kXG4Bary[q][1], a ) * std::pow( kXG4Bary[q][2], bb ) * std::pow( kXG4Bary[q][3], c );
            b[row] = fact( a ) * fact( bb ) * fact( c ) / fact( a + bb + c + 3 );
         }
   for ( int k = 0; k < n; ++k )
   {
      double nrm = 0;
      for ( int i = k; i < m; ++i ) nrm += A[i * n + k] * A[i * n + k];
      nrm = std::sqrt( nrm );
      const double alpha = A[k * n + k] > 0 ? -nrm : nrm;
      std::vector< double > v( m, 0.0 );
      for ( int i = k; i < m; ++i ) v[i] = A[i * n + k];
      v[k] -= alpha;
      double vv = 0;
      for ( int i = k; i < m; ++i ) vv += v[i] * v[i];
      if ( vv == 0 ) continue;
      for ( int j = k; j < n; ++j )
      {
         double d = 0;
         for ( int i = k; i < m; ++i ) d += v[i] * A[i * n + j];
         for ( int i = k; i < m; ++i ) A[i * n + j] -= 2 * d / vv * v[i];
      }
      double d = 0;
      for ( int i = k; i < m; ++i ) d += v[i] * b[i];
      for ( int i = k; i < m; ++i ) b[i] -= 2 * d / vv * v[i];
   }
   for ( int k = n - 1; k >= 0; --k )
   {
      double s = b[k];
      for ( int j = k + 1; j < n; ++j ) s -= A[k * n + j] * w[j];
      w[k] = s / A[k * n + k];
   }
}

void ensure_p2_constants()
{
   static PerDeviceOnce once;
   once.run( [] {
      double pts[11][3], w[11], g[11][10][3];
      xg4_weights( w );
      const double lg[4][3] = { { -1, -1, -1 }, { 1, 0, 0 }, { 0, 1, 0 }, { 0, 0, 1 } };
      const int    ed[6][2] = { { 2, 3 }, { 1, 3 }, { 1, 2 }, { 0, 3 }, { 0, 2 }, { 0, 1 } };
      for ( int q = 0; q < 11; ++q )
      {
         for ( int d = 0; d < 3; ++d ) pts[q][d] = kXG4Bary[q][d + 1];
         const double lam[4] = { 1.0 - pts[q][0] - pts[q][1] - pts[q][2], pts[q][0], pts[q][1], pts[q][2] };
         for ( int i = 0; i < 4; ++i )
            for ( int d = 0; d < 3; ++d ) g[q][i][d] = ( 4.0 * lam[i] - 1.0 ) * lg[i][d];
         for ( int e = 0; e < 6; ++e )
            for ( int d = 0; d < 3; ++d )
               g[q][4 + e][d] = 4.0 * ( lam[ed[e][0]] * lg[ed[e][1]][d] + lam[ed[e][1]] * lg[ed[e][0]][d] );
      }
      check_cuda( cudaMemcpyToSymbol( c_xg4_pts, pts, sizeof( pts ) ), "P2 constants (points)" );
      double bary[11][4];
      for ( int q = 0; q < 11; ++q )
      {
         bary[q][0] = 1.0 - pts[q][0] - pts[q][1] - pts[q][2];
         for ( int d = 0; d < 3; ++d ) bary[q][d + 1] = pts[q][d];
      }
      check_cuda( cudaMemcpyToSymbol( c_xg4_bary, bary, sizeof( bary ) ), "P2 constants (barycentric points)" );
      double mass[11][10];
      for ( int q = 0; q < 11; ++q )
         for ( int i = 0, v = 0; i < 4; ++i )
            for ( int j = i; j < 4; ++j, ++v ) mass[q][v] = w[q] * bary[q][i] * bary[q][j];
      check_cuda( cudaMemcpyToSymbol( c_xg4_mass, mass, sizeof( mass ) ), "P2 constants (products)" );
      int8_t loc[6][10];
      for ( int ty = 0; ty < 6; ++ty )
         for ( int i = 0; i < 10; ++i )
            loc[ty][i] = int8_t( p2_local( ty, i, 0 ) + 3 * p2_local( ty, i, 1 ) + 9 * p2_local( ty, i, 2 ) );

      check_cuda( cudaMemcpyToSymbol( c_p2_loc, loc, sizeof( loc ) ), "P2 constants (local nodes)" );
      int8_t node0[27];
      for ( int l = 0; l < 27; ++l ) node0[l] = -1;
      for ( int i = 0; i < 10; ++i ) node0[loc[0][i]] = int8_t( i );
      check_cuda( cudaMemcpyToSymbol( c_p2_node0, node0, sizeof( node0 ) ), "P2 constants (local nodes)" );
      int8_t from[60], from0[28];
      int    nf = 0;
      for ( int l = 0; l < 27; ++l )
      {
         from0[l] = int8_t( nf );
         for ( int v = 0; v < 60; ++v )
            if ( loc[v / 10][v % 10] == l ) from[nf++] = int8_t( v );
      }
      from0[27] = int8_t( nf );
      check_cuda( cudaMemcpyToSymbol( c_p2_from, from, sizeof( from ) ), "P2 constants (node sums)" );
      check_cuda( cudaMemcpyToSymbol( c_p2_from0, from0, sizeof( from0 ) ), "P2 constants (node sums)" );
      check_cuda( cudaMemcpyToSymbol( c_xg4_w, w, sizeof( w ) ), "P2 constants (weights)" );
      check_cuda( cudaMemcpyToSymbol( c_p2_rgrad, g, sizeof( g ) ), "P2 constants (gradients)" );
      double phi[11][10];
      for ( int q = 0; q < 11; ++q )
      {
         const double lam[4] = { 1.0 - pts[q][0] - pts[q][1] - pts[q][2], pts[q][0], pts[q][1], pts[q][2] };
         for ( int i = 0; i < 4; ++i ) phi[q][i] = lam[i] * ( 2.0 * lam[i] - 1.0 );
         for ( int e = 0; e < 6; ++e ) phi[q][4 + e] = 4.0 * lam[ed[e][0]] * lam[ed[e][1]];
      }
      check_cuda( cudaMemcpyToSymbol( c_p2_phi, phi, sizeof( phi ) ), "P2 constants (basis values)" );
      int8_t ent[600];
      p2_stored_entries( ent );
      check_cuda( cudaMemcpyToSymbol( c_p2s_ent, ent, sizeof( ent ) ), "P2 constants (stencil entries)" );
   } );
}

// ---------------------------------------------------------------------------------------------
// Matrix-free P2 passes: what a quadrature point needs
//
// On a micro-cell J is constant, so only the blending map's DF varies between points.  For the shell
// DF = s I + X g^T (s = R / |X|, g the gradient of s), a rank-one update, so
//    det DF = s^2 m,  DF^-1 = (I - X g^T / m) / s,  DF^-T = (I - g X^T / m) / s,  m = s + g . X,
// and R's weight t = t0 + sum_k lambda_k(q) t_k is affine too.  Gradients of quadratic functions are affine,
// so they are interpolated from the four vertices: grad u at vertex k is a combination of ten node
// values with integer weights, and sum_q of the pairing with every basis gradient needs only
// H_k = sum_q lambda_k(q) h(q) at the four vertices.  Per point this takes about 100 operations and the
// coefficient, against 300 for the 3x3 inverse and two loops over ten reference gradients.
//
// What a micro-cell computes once (J, its inverse, t, the gradients at the vertices and the final pairing)
// is computed in FP64 for every value type, and only the loop over the points in the accumulation type: the
// vertices' gradients cancel at the points and J is a difference of coordinates, so that in FP32 the whole
// was less exact than evaluating every point by itself.
// ---------------------------------------------------------------------------------------------
template < typename A >
struct ShellPoint {
   A X[3], g[3];
   A s, m, im, R;
};

__device__ __forceinline__ double rsqrt_of( double v ) { return rsqrt( v ); }
__device__ __forceinline__ float  rsqrt_of( float v ) { return rsqrtf( v ); }

// one micro-cell of an anchor: first vertex, columns of J, J^-1, |det J| and the shell map's weight t at the
// first vertex and its differences to the others (A: type of the points; J^-1 and |det J| in FP64)
template < typename A >
struct MicroCell {
   A      X0[3], J[3][3];
   A      t[4];
   A      bx[3], rad, dr;  // gradient of t; R = rad + |t| dr
   double Ji[3][3], adet;
};

template < typename A >
__device__ __forceinline__ void micro_cell( const CellGeom& g, int ne, int ty, int x, int y, int z, MicroCell< A >& c )
{
   const double inv_n = 1.0 / double( ne ), v0[3] = { double( x + c_mc_off[ty][0][0] ), double( y + c_mc_off[ty][0][1] ), double( z + c_mc_off[ty][0][2] ) };
   const double iv    = g.blend == 1 ? 1.0 / g.volT : 0.0;
   double       J[3][3], t[4] = { 0, 0, 0, 0 };
   for ( int d = 0; d < 3; ++d )
   {
      double st[3];  // computational steps
      for ( int k = 0; k < 3; ++k ) st[k] = ( g.P[k + 1][d] - g.P[0][d] ) * inv_n;
      const double X = g.P[0][d] + st[0] * v0[0] + st[1] * v0[1] + st[2] * v0[2], b = g.bxc[d] * iv;
      for ( int k = 0; k < 3; ++k )
      {
         J[d][k] = st[0] * double( c_mc_off[ty][k + 1][0] - c_mc_off[ty][0][0] ) + st[1] * double( c_mc_off[ty][k + 1][1] - c_mc_off[ty][0][1] ) +
                   st[2] * double( c_mc_off[ty][k + 1][2] - c_mc_off[ty][0][2] );
         c.J[d][k] = A( J[d][k] );
         t[k + 1] += b * J[d][k];
      }
      t[0] += b * ( X - g.ray[d] );
      c.X0[d] = A( X );
      c.bx[d] = A( b );
   }
   for ( int k = 0; k < 4; ++k ) c.t[k] = A( t[k] );
   c.rad = A( g.rad_ray );
   c.dr  = A( g.rad_ref - g.rad_ray );
   const double c0 = J[1][1] * J[2][2] - J[1][2] * J[2][1], c1 = J[1][2] * J[2][0] - J[1][0] * J[2][2], c2 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
   const double det = J[0][0] * c0 + J[0][1] * c1 + J[0][2] * c2, id = 1.0 / det;
   c.Ji[0][0] = c0 * id;
   c.Ji[1][0] = c1 * id;
   c.Ji[2][0] = c2 * id;
   c.Ji[0][1] = ( J[0][2] * J[2][1] - J[0][1] * J[2][2] ) * id;
   c.Ji[1][1] = ( J[0][0] * J[2][2] - J[0][2] * J[2][0] ) * id;
   c.Ji[2][1] = ( J[0][1] * J[2][0] - J[0][0] * J[2][1] ) * id;
   c.Ji[0][2] = ( J[0][1] * J[1][2] - J[0][2] * J[1][1] ) * id;
   c.Ji[1][2] = ( J[0][2] * J[1][0] - J[0][0] * J[1][2] ) * id;
   c.Ji[2][2] = ( J[0][0] * J[1][1] - J[0][1] * J[1][0] ) * id;
   c.adet     = fabs( det );
}

// point of barycentric weights l1, l2, l3 and the shell map there
template < typename A >
__device__ __forceinline__ void cell_point( const MicroCell< A >& c, A l1, A l2, A l3, ShellPoint< A >& p )
{
#pragma unroll
   for ( int d = 0; d < 3; ++d ) p.X[d] = c.X0[d] + c.J[d][0] * l1 + c.J[d][1] * l2 + c.J[d][2] * l3;
}
template < typename A >
__device__ __forceinline__ void shell_point( const MicroCell< A >& c, A l1, A l2, A l3, ShellPoint< A >& p )
{
   const A t  = c.t[0] + c.t[1] * l1 + c.t[2] * l2 + c.t[3] * l3;
   p.R        = c.rad + fabs( t ) * c.dr;
   const A d  = t < A( 0 ) ? -c.dr : c.dr;
   const A ir = rsqrt_of( p.X[0] * p.X[0] + p.X[1] * p.X[1] + p.X[2] * p.X[2] );
   p.s        = p.R * ir;
   const A e  = ir * d, f = p.s * ir * ir;
   for ( int k = 0; k < 3; ++k ) p.g[k] = e * c.bx[k] - f * p.X[k];
   p.m  = p.s + ( p.g[0] * p.X[0] + p.g[1] * p.X[1] + p.g[2] * p.X[2] );
   p.im = A( 1 ) / p.m;
}

// gradients of the quadratic function with node values u at the four vertices, with respect to X
template < typename A >
__device__ __forceinline__ void p2_vertex_gradients( const A u_[10], const double Ji[3][3], A G[4][3] )
{
   double u[10];
#pragma unroll
   for ( int i = 0; i < 10; ++i ) u[i] = double( u_[i] );
   // c[k][l]: coefficient of grad lambda_l at vertex k
   const double c[4][4] = { { 3 * u[0], 4 * u[9] - u[1], 4 * u[8] - u[2], 4 * u[7] - u[3] },
                            { 4 * u[9] - u[0], 3 * u[1], 4 * u[6] - u[2], 4 * u[5] - u[3] },
                            { 4 * u[8] - u[0], 4 * u[6] - u[1], 3 * u[2], 4 * u[4] - u[3] },
                            { 4 * u[7] - u[0], 4 * u[5] - u[1], 4 * u[4] - u[2], 3 * u[3] } };
#pragma unroll
   for ( int k = 0; k < 4; ++k )
   {
      const double r0 = c[k][1] - c[k][0], r1 = c[k][2] - c[k][0], r2 = c[k][3] - c[k][0];
#pragma unroll
      for ( int d = 0; d < 3; ++d ) G[k][d] = A( r0 * Ji[0][d] + r1 * Ji[1][d] + r2 * Ji[2][d] );
   }
}

// the transpose: y[i] = sum_k (gradient of basis function i at vertex k) . H[k]
template < typename A >
__device__ __forceinline__ void p2_pair_gradients( const A H[4][3], const double Ji[3][3], A y[10] )
{
   double h[4][4];
#pragma unroll
   for ( int k = 0; k < 4; ++k )
   {
      const double a = double( H[k][0] ), b = double( H[k][1] ), c = double( H[k][2] );
#pragma unroll
      for ( int d = 0; d < 3; ++d ) h[k][d + 1] = Ji[d][0] * a + Ji[d][1] * b + Ji[d][2] * c;
      h[k][0] = -( h[k][1] + h[k][2] + h[k][3] );
   }
#pragma unroll
   for ( int i = 0; i < 4; ++i ) y[i] = A( 4 * h[i][i] - ( ( h[0][i] + h[1][i] ) + ( h[2][i] + h[3][i] ) ) );
   y[4] = A( 4 * ( h[2][3] + h[3][2] ) );
   y[5] = A( 4 * ( h[1][3] + h[3][1] ) );
   y[6] = A( 4 * ( h[1][2] + h[2][1] ) );
   y[7] = A( 4 * ( h[0][3] + h[3][0] ) );
   y[8] = A( 4 * ( h[0][2] + h[2][0] ) );
   y[9] = A( 4 * ( h[0][1] + h[1][0] ) );
}

// the coefficient at point q of a micro-cell: from its node values kl (NODAL) or the closed form at F
template < typename A, bool NODAL >
__device__ __forceinline__ A p2_coefficient( const Coefficient& kc, int q, const A* kl, const A* F, A radius )
{
   if constexpr ( NODAL )
   {
      A kq = A( 0 );
#pragma unroll
      for ( int i = 0; i < 10; ++i ) kq += A( c_p2_phi[q][i] ) * kl[i];
      return kq;
   }
   else
      return coeff_eval( kc, F, radius );
}

// K u of one micro-cell: node values u in, sums y out (kl: the coefficient's node values, NODAL only)
template < typename A, bool NODAL, bool BLEND >
__device__ __forceinline__ void p2_micro_apply( const CellGeom& g, const Coefficient& kc, int ne, int ty, int x, int y, int z,
                                                const A u[10], const A* kl, A yl[10] )
{
   MicroCell< A > mc;
   micro_cell( g, ne, ty, x, y, z, mc );
   if constexpr ( !BLEND )
   {
      // J is all there is, so H_k = sum_j M_kj G_j with M_kj = sum_q w k lambda_k lambda_j: ten sums per point
      double M[10];
#pragma unroll
      for ( int v = 0; v < 10; ++v ) M[v] = 0;
#pragma unroll 1
      for ( int q = 0; q < 11; ++q )
      {
         ShellPoint< A > p;
         cell_point( mc, A( c_xg4_bary[q][1] ), A( c_xg4_bary[q][2] ), A( c_xg4_bary[q][3] ), p );
         const double f = double( p2_coefficient< A, NODAL >( kc, q, kl, p.X, A( -1 ) ) );
#pragma unroll
         for ( int v = 0; v < 10; ++v ) M[v] += f * c_xg4_mass[q][v];
      }
      double G[4][3], H[4][3], ud[10], yd[10];
#pragma unroll
      for ( int i = 0; i < 10; ++i ) ud[i] = double( u[i] );
      p2_vertex_gradients( ud, mc.Ji, G );
#pragma unroll
      for ( int k = 0; k < 4; ++k )
#pragma unroll
         for ( int d = 0; d < 3; ++d )
         {
            H[k][d] = 0;
#pragma unroll
            for ( int j = 0; j < 4; ++j )
            {
               const int lo = k < j ? k : j, hi = k < j ? j : k;
               H[k][d] += M[lo * 4 - lo * ( lo - 1 ) / 2 + ( hi - lo )] * G[j][d];
            }
         }
      p2_pair_gradients( H, mc.Ji, yd );
#pragma unroll
      for ( int i = 0; i < 10; ++i ) yl[i] = A( yd[i] * mc.adet );
      return;
   }
   A G[4][3], H[4][3];
   p2_vertex_gradients( u, mc.Ji, G );
#pragma unroll
   for ( int k = 0; k < 4; ++k ) H[k][0] = H[k][1] = H[k][2] = A( 0 );
   // rolled: the body is about 400 instructions, and eleven copies cost more in instruction fetches than
   // the constants of the points save (3.18 against 2.67 ms on the shell of k_p2_apply_pass with blocks of 96)
#pragma unroll 1
   for ( int q = 0; q < 11; ++q )
   {
      const A l0 = A( c_xg4_bary[q][0] ), l1 = A( c_xg4_bary[q][1] ), l2 = A( c_xg4_bary[q][2] ), l3 = A( c_xg4_bary[q][3] );
      A       B[3], F[3];
#pragma unroll
      for ( int d = 0; d < 3; ++d ) B[d] = l0 * G[0][d] + l1 * G[1][d] + l2 * G[2][d] + l3 * G[3][d];
      ShellPoint< A > p;
      cell_point( mc, l1, l2, l3, p );
      // |det DF| DF^-1 DF^-T B = |m| (w - X (g . w) / m),  w = B - g (X . B) / m
      shell_point( mc, l1, l2, l3, p );
      const A xb = ( p.X[0] * B[0] + p.X[1] * B[1] + p.X[2] * B[2] ) * p.im;
#pragma unroll
      for ( int d = 0; d < 3; ++d ) B[d] -= p.g[d] * xb;
      const A gw = ( p.g[0] * B[0] + p.g[1] * B[1] + p.g[2] * B[2] ) * p.im;
#pragma unroll
      for ( int d = 0; d < 3; ++d )
      {
         B[d] -= p.X[d] * gw;
         F[d] = p.X[d] * p.s;
      }
      const A f = A( c_xg4_w[q] * mc.adet ) * fabs( p.m ) * p2_coefficient< A, NODAL >( kc, q, kl, F, p.R );
#pragma unroll
      for ( int d = 0; d < 3; ++d )
      {
         const A h = f * B[d];
         H[0][d] += l0 * h;
         H[1][d] += l1 * h;
         H[2][d] += l2 * h;
         H[3][d] += l3 * h;
      }
   }
   p2_pair_gradients( H, mc.Ji, yl );
}

// y += K x of one parity pass, matrix-free (anchors of one parity share no node, see k_p2_pass).  Bound
// by the latency and rate of FP64 arithmetic, three quarters of it the coefficient and the map.
//
// A thread takes one anchor and keeps the 27 nodes its six micro-cells touch in shared memory (values in,
// sums out), so that global memory sees each of them once per pass, all loads in flight together, instead
// of ten read-modify-writes per micro-cell in a chain.  Anchors at the slanted face have one micro-cell and
// work straight from global memory.  Blocks run over (cell, anchor) of one kind (six, five or one
// micro-cells), so they are full whatever the number of anchors per cell and a warp's threads do the same
// work.
//
// Shell of 1920 macro-cells, level 4 (7.9 M micro-cells), exp/sin coefficient, per apply: 6.22 ms with a
// 3x3 inverse per point and chained updates, 2.24 ms so (64 threads, 168 registers; with 96 threads 1 %, with
// 128 registers 18 %, with two points at a time 2 % more).
constexpr int kP2ApplyThreads = 64;
template < typename T, typename A, bool NODAL, bool BLEND >
__global__ void __launch_bounds__( kP2ApplyThreads, 6 )
    k_p2_apply_pass( int ne, int nC, int3 kinds, int3 blocks, const int* __restrict__ anch, const int64_t* __restrict__ cell_off,
                     const CellGeom* __restrict__ geom, Coefficient kc, const T* __restrict__ src, A* __restrict__ acc,
                     int64_t level_size, int* err, const double* __restrict__ kn )
{
   extern __shared__ __align__( 16 ) unsigned char p2_raw[];
   A* const  xs = reinterpret_cast< A* >( p2_raw ) + threadIdx.x;  // node l of this thread: xs[l * kP2ApplyThreads]
   A* const  ys = xs + 27 * kP2ApplyThreads;
   const int ns = 2 * ne;
   int       bk = blockIdx.x, n = kinds.x, first = 0;
   if ( bk >= blocks.x )
   {
      bk -= blocks.x, first = kinds.x, n = kinds.y;
      if ( bk >= blocks.y ) bk -= blocks.y, first += kinds.y, n = 0;
   }
   const bool     single = n == 0;
   const unsigned per    = unsigned( single ? kinds.z : n );
   const int64_t  t      = int64_t( bk ) * kP2ApplyThreads + threadIdx.x;
   if ( t >= int64_t( nC ) * per ) return;
   const int      c    = t < 0x7fffffff ? int( unsigned( t ) / per ) : int( t / per );
   const int      a    = anch[first + int( t - int64_t( c ) * per )];
   const int      x = a & 1023, y = ( a >> 10 ) & 1023, z = a >> 20, room = ns - 2 * ( x + y + z );
   const int64_t  base = cell_off[c];
   {
      // self-check: every node of the window inside the level's vector
      const int64_t last = base + window_last( ns, 2 * x, 2 * y, 2 * z, 2, room );
      if ( room < 2 || base < 0 || last >= level_size )
      {
         atomicExch( err, 2 );
         return;
      }
   }
   auto at = [&]( int l ) { return base + cidx( ns, 2 * x + l % 3, 2 * y + ( l / 3 ) % 3, 2 * z + l / 9 ); };
   if ( single )
   {
      A       u[10], kl[NODAL ? 10 : 1], yl[10];
      int64_t i0[10];
#pragma unroll
      for ( int i = 0; i < 10; ++i )
      {
         i0[i] = at( c_p2_loc[0][i] );
         u[i]  = A( ld_any( src + i0[i] ) );
         if constexpr ( NODAL ) kl[i] = A( kn[i0[i]] );
      }
      p2_micro_apply< A, NODAL, BLEND >( geom[c], kc, ne, 0, x, y, z, u, kl, yl );
#pragma unroll
      for ( int i = 0; i < 10; ++i ) acc[i0[i]] += yl[i];
      return;
   }
#pragma unroll
   for ( int r = 0; r < 9; ++r )
   {
      const int64_t row = at( 3 * r );
#pragma unroll
      for ( int k = 0; k < 3; ++k )
      {
         xs[( 3 * r + k ) * kP2ApplyThreads] = k + r % 3 + r / 3 <= room ? A( ld_any( src + row + k ) ) : A( 0 );
         ys[( 3 * r + k ) * kP2ApplyThreads] = A( 0 );
      }
   }
#pragma unroll 1
   for ( int ty = 0; ty < 6; ++ty )
   {
      if ( x + y + z > ne - 1 - c_mc_shift[ty] ) continue;
      A u[10], kl[NODAL ? 10 : 1], yl[10];
#pragma unroll
      for ( int i = 0; i < 10; ++i )
      {
         u[i] = xs[c_p2_loc[ty][i] * kP2ApplyThreads];
         if constexpr ( NODAL ) kl[i] = A( kn[at( c_p2_loc[ty][i] )] );
      }
      p2_micro_apply< A, NODAL, BLEND >( geom[c], kc, ne, ty, x, y, z, u, kl, yl );
#pragma unroll
      for ( int i = 0; i < 10; ++i ) ys[c_p2_loc[ty][i] * kP2ApplyThreads] += yl[i];
   }
#pragma unroll
   for ( int r = 0; r < 9; ++r )
   {
      const int64_t row = at( 3 * r );
#pragma unroll
      for ( int k = 0; k < 3; ++k )
         if ( k + r % 3 + r / 3 <= room ) acc[row + k] += ys[( 3 * r + k ) * kP2ApplyThreads];
   }
}

// The same pass with one thread per micro-cell, for levels whose classes hold fewer anchors than the pass
// above keeps in flight (there it takes the time of one thread's six micro-cells, 60 us a pass, however
// small the level): warp w of a block takes type w of 32 anchors, whose nodes the block shares; their
// sums are added in a fixed order.  Anchors with one micro-cell are taken one per thread, straight from
// global memory (their blocks would hold one busy warp in six).
constexpr int kP2SplitThreads = 192;
template < typename T, typename A, bool NODAL, bool BLEND >
__global__ void __launch_bounds__( kP2SplitThreads, 3 )
    k_p2_apply_split( int ne, int nC, int3 kinds, int3 blocks, const int* __restrict__ anch, const int64_t* __restrict__ cell_off,
                     const CellGeom* __restrict__ geom, Coefficient kc, const T* __restrict__ src, A* __restrict__ acc,
                     int64_t level_size, int* err, const double* __restrict__ kn )
{
   __shared__ A xs[27][32], ys[60][32], ks[NODAL ? 27 : 1][32];
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ns = 2 * ne;
   // the block's anchors: kind, first one among (cell, anchor) of the kind
   int bk = blockIdx.x, n = kinds.x, first = 0;
   if ( bk >= blocks.x )
   {
      bk -= blocks.x, first = kinds.x, n = kinds.y;
      if ( bk >= blocks.y ) bk -= blocks.y, first += kinds.y, n = 0;
   }
   const bool     single = n == 0;
   const unsigned per    = unsigned( single ? kinds.z : n );
   const int64_t  t      = single ? int64_t( bk ) * kP2SplitThreads + threadIdx.x : int64_t( bk ) * 32 + lane;
   bool           live   = t < int64_t( nC ) * per;
   const int64_t  tt     = live ? t : 0;
   const int      c      = tt < 0x7fffffff ? int( unsigned( tt ) / per ) : int( tt / per );
   const int      a      = anch[first + int( tt - int64_t( c ) * per )];
   const int      x = a & 1023, y = ( a >> 10 ) & 1023, z = a >> 20, room = ns - 2 * ( x + y + z );
   const int64_t  base = cell_off[c];
   {
      // self-check: every node of the window inside the level's vector
      const int64_t last = base + window_last( ns, 2 * x, 2 * y, 2 * z, 2, room );
      if ( live && ( room < 2 || base < 0 || last >= level_size ) )
      {
         atomicExch( err, 2 );
         live = false;
      }
   }
   if ( single )
   {
      if ( !live ) return;
      A       u[10], kl[NODAL ? 10 : 1], yl[10];
      int64_t at[10];
#pragma unroll
      for ( int i = 0; i < 10; ++i )
      {
         const int l = c_p2_loc[0][i];
         at[i]       = base + cidx( ns, 2 * x + l % 3, 2 * y + ( l / 3 ) % 3, 2 * z + l / 9 );
         u[i]        = A( ld_any( src + at[i] ) );
         if constexpr ( NODAL ) kl[i] = A( kn[at[i]] );
      }
      p2_micro_apply< A, NODAL, BLEND >( geom[c], kc, ne, 0, x, y, z, u, kl, yl );
#pragma unroll
      for ( int i = 0; i < 10; ++i ) acc[at[i]] += yl[i];
      return;
   }
   // node a + 3 b + 9 c of the window, if it exists
   auto node = [&]( int l, int64_t& at ) -> bool {
      const int da = l % 3, db = ( l / 3 ) % 3, dc = l / 9;
      at           = base + cidx( ns, 2 * x + da, 2 * y + db, 2 * z + dc );
      return live && da + db + dc <= room;
   };
#pragma unroll
   for ( int r = 0; r < 5; ++r )
   {
      const int l = warp + 6 * r;
      int64_t   at;
      if ( l < 27 )
      {
         const bool in = node( l, at );
         xs[l][lane]   = in ? A( ld_any( src + at ) ) : A( 0 );
         if constexpr ( NODAL ) ks[l][lane] = in ? A( kn[at] ) : A( 0 );
      }
   }
   __syncthreads();
   if ( live && x + y + z <= ne - 1 - c_mc_shift[warp] )
   {
      A u[10], kl[NODAL ? 10 : 1], yl[10];
#pragma unroll
      for ( int i = 0; i < 10; ++i )
      {
         u[i] = xs[c_p2_loc[warp][i]][lane];
         if constexpr ( NODAL ) kl[i] = ks[c_p2_loc[warp][i]][lane];
      }
      p2_micro_apply< A, NODAL, BLEND >( geom[c], kc, ne, warp, x, y, z, u, kl, yl );
#pragma unroll
      for ( int i = 0; i < 10; ++i ) ys[10 * warp + i][lane] = yl[i];
   }
   else
#pragma unroll
      for ( int i = 0; i < 10; ++i ) ys[10 * warp + i][lane] = A( 0 );
   __syncthreads();
#pragma unroll
   for ( int r = 0; r < 5; ++r )
   {
      const int l = warp + 6 * r;
      int64_t   at;
      if ( l < 27 && node( l, at ) )
      {
         A s = A( 0 );
         for ( int k = c_p2_from0[l]; k < c_p2_from0[l + 1]; ++k ) s += ys[c_p2_from[k]][lane];
         acc[at] += s;
      }
   }
}

// mapped quantities of quadrature point q of a micro-cell: Mi = (DF J)^-1 and s = w k |det(DF J)|
// kl: the coefficient's values at the ten nodes (a coefficient stored as a P2 function), or nullptr
// for the closed form at the blended point
template < typename A >
__device__ __forceinline__ void p2_point( const CellGeom& g, const Coefficient& kc, const A X0[3], const A J[3][3], int q, A Mi[3][3],
                                          A& s, const A* kl )
{
   A Xq[3];
   for ( int r = 0; r < 3; ++r )
      Xq[r] = X0[r] + J[r][0] * A( c_xg4_pts[q][0] ) + J[r][1] * A( c_xg4_pts[q][1] ) + J[r][2] * A( c_xg4_pts[q][2] );
   A M[3][3], Fq[3];
   if ( g.blend == 1 )
   {
      A DF[3][3];
      shell_map( g, Xq, Fq, DF );
      for ( int r = 0; r < 3; ++r )
         for ( int c = 0; c < 3; ++c ) M[r][c] = DF[r][0] * J[0][c] + DF[r][1] * J[1][c] + DF[r][2] * J[2][c];
   }
   else
      for ( int r = 0; r < 3; ++r )
      {
         Fq[r] = Xq[r];
         for ( int c = 0; c < 3; ++c ) M[r][c] = J[r][c];
      }
   const A c00 = M[1][1] * M[2][2] - M[1][2] * M[2][1];
   const A c01 = M[1][2] * M[2][0] - M[1][0] * M[2][2];
   const A c02 = M[1][0] * M[2][1] - M[1][1] * M[2][0];
   const A det = M[0][0] * c00 + M[0][1] * c01 + M[0][2] * c02;
   const A id  = A( 1 ) / det;
   Mi[0][0]    = c00 * id;
   Mi[1][0]    = c01 * id;
   Mi[2][0]    = c02 * id;
   Mi[0][1]    = ( M[0][2] * M[2][1] - M[0][1] * M[2][2] ) * id;
   Mi[1][1]    = ( M[0][0] * M[2][2] - M[0][2] * M[2][0] ) * id;
   Mi[2][1]    = ( M[0][1] * M[2][0] - M[0][0] * M[2][1] ) * id;
   Mi[0][2]    = ( M[0][1] * M[1][2] - M[0][2] * M[1][1] ) * id;
   Mi[1][2]    = ( M[0][2] * M[1][0] - M[0][0] * M[1][2] ) * id;
   Mi[2][2]    = ( M[0][0] * M[1][1] - M[0][1] * M[1][0] ) * id;
   A kq;
   if ( kl )
   {
      kq = A( 0 );
      for ( int i = 0; i < 10; ++i ) kq += A( c_p2_phi[q][i] ) * kl[i];
   }
   else
      kq = coeff_eval( kc, Fq );
   s = A( c_xg4_w[q] ) * kq * fabs( det );
}

// physical gradient of basis function i at point q: row (reference gradient) times Mi
template < typename A >
__device__ __forceinline__ void p2_grad( int q, int i, const A Mi[3][3], A G[3] )
{
   for ( int d = 0; d < 3; ++d )
      G[d] = A( c_p2_rgrad[q][i][0] ) * Mi[0][d] + A( c_p2_rgrad[q][i][1] ) * Mi[1][d] + A( c_p2_rgrad[q][i][2] ) * Mi[2][d];
}

// One parity pass over the level-L micro-cells (anchors of parity (px, py, pz); ne = 2^L), nodes on
// storage level L+1.  MODE 1: diagonal of K into acc; 2: K added to the assembled stencils of its nodes
// (st, layout of sv, whose macro-cells are the launch's: first_cell and those after it).  Anchors of one parity share no node, and the micro-cells of one anchor are taken in
// order by one thread, so plain additions are deterministic.
template < typename A, int MODE >
__global__ void __launch_bounds__( 256, 2 ) k_p2_pass( int ne, int first_cell, int nanch, const int* __restrict__ anch, const int64_t* __restrict__ cell_off,
                                                       const CellGeom* __restrict__ geom, Coefficient kc, A* __restrict__ acc,
                                                       P2StoredView sv, A* __restrict__ st, int64_t st_size, int64_t level_size, int* err,
                                                       const double* __restrict__ kn )
{
   const int t = blockIdx.x * blockDim.x + threadIdx.x;  // one micro-cell anchor per thread
   const int c = first_cell + int( blockIdx.y );
   if ( t >= nanch ) return;
   const int      a = anch[t];
   const int      x = a & 1023, y = ( a >> 10 ) & 1023, z = a >> 20, ns = 2 * ne;
   const CellGeom g    = geom[c];
   const int64_t  base = cell_off[c];
   for ( int ty = 0; ty < 6; ++ty )
   {
      if ( x + y + z > ne - 1 - c_mc_shift[ty] ) continue;
      MicroCell< A > mc;
      micro_cell( g, ne, ty, x, y, z, mc );
      int64_t idx[10];
      A       kl[10];
      bool    bad = false;
      for ( int m = 0; m < 10; ++m )
      {
         const int l = c_p2_loc[ty][m];
         idx[m]      = base + cidx( ns, 2 * x + l % 3, 2 * y + ( l / 3 ) % 3, 2 * z + l / 9 );
         bad |= idx[m] < 0 || idx[m] >= level_size;
      }
      // self-check: nodes inside the level's vector
      if ( bad )
      {
         atomicExch( err, 2 );
         continue;
      }
      if ( kn )
         for ( int m = 0; m < 10; ++m ) kl[m] = A( kn[idx[m]] );
      A K[MODE == 2 ? 55 : 10];
      for ( int v = 0; v < ( MODE == 2 ? 55 : 10 ); ++v ) K[v] = A( 0 );
#pragma unroll 1
      for ( int q = 0; q < 11; ++q )
      {
         A Mi[3][3], s;
         p2_point( g, kc, mc.X0, mc.J, q, Mi, s, kn ? kl : static_cast< const A* >( nullptr ) );
         if constexpr ( MODE == 1 )
            for ( int i = 0; i < 10; ++i )
            {
               A G[3];
               p2_grad( q, i, Mi, G );
               K[i] += s * ( G[0] * G[0] + G[1] * G[1] + G[2] * G[2] );
            }
         else
         {
            A G[10][3];
            for ( int i = 0; i < 10; ++i ) p2_grad( q, i, Mi, G[i] );
            int v = 0;
            for ( int i = 0; i < 10; ++i )
               for ( int j = i; j < 10; ++j, ++v ) K[v] += s * ( G[i][0] * G[j][0] + G[i][1] * G[j][1] + G[i][2] * G[j][2] );
         }
      }
      if constexpr ( MODE == 1 )
         for ( int i = 0; i < 10; ++i ) acc[idx[i]] += K[i];
      else
#pragma unroll
         for ( int i = 0; i < 10; ++i )
         {
            const int     l = c_p2_loc[ty][i];
            int64_t       skip;
            const int64_t w = p2_weight_at( sv, int( blockIdx.y ), 2 * x + l % 3, 2 * y + ( l / 3 ) % 3, 2 * z + l / 9, skip );
#pragma unroll
            for ( int j = 0; j < 10; ++j )
            {
               const int     lo = i < j ? i : j, hi = i < j ? j : i;
               const int64_t at = w + c_p2s_ent[( 10 * ty + i ) * 10 + j] * skip;
               // self-check: stored weights inside their array
               if ( at < 0 || at >= st_size ) atomicExch( err, 2 );
               else st[at] += K[lo * 10 - lo * ( lo - 1 ) / 2 + ( hi - lo )];
            }
         }
   }
}

// Combine: cell interior points take s = acc, face/edge/vertex owners the sum of their copies in
// the neighbouring cells; then the operation's epilogue (the constant-stencil kernels' semantics).
template < typename T, typename A, int OP >
__device__ __forceinline__ A epilogue_value( int64_t i, A s, A invd, const T* src, const T* v1, T* v2, A a0, A a1, A* second )
{
   if constexpr ( OP == OP_APPLY || OP == OP_APPLY_ADD ) return s;
   else if constexpr ( OP == OP_RESID ) return A( ld_any( v1 + i ) ) - s;
   else if constexpr ( OP == OP_JAC ) return A( ld_any( src + i ) ) + a0 * ( invd * ( A( ld_any( v1 + i ) ) - s ) );
   else if constexpr ( OP == OP_CHEB0 ) return invd * ( A( ld_any( v1 + i ) ) - s );
   else if constexpr ( OP == OP_CHEBI )
   {
      *second = A( ld_any( v2 + i ) ) + a0 * A( ld_any( src + i ) );
      return invd * s;
   }
   else if constexpr ( OP == OP_CHEBL ) return ( A( ld_any( v2 + i ) ) + a0 * A( ld_any( src + i ) ) ) + a1 * ( invd * s );
   else if constexpr ( OP == OP_DINV_APPLY ) return invd * s;
   return s;
}

// the vectors of up to three components that one combine launch serves
template < typename T, typename A >
struct AccVecs {
   const A* acc[3];
   const T* src[3];
   const T* v1[3];
   T*       v2[3];
   T*       dst[3];
};

// cell interiors of one component (blockIdx.y): the listed points, one thread each, on levels that list
// them, else a warp per row
// (the component is selected by comparison: indexing a kernel parameter with a runtime value copies it to local memory)
template < typename P >
__device__ __forceinline__ P component( const P ( &v )[3], unsigned k )
{
   return k == 0 ? v[0] : k == 1 ? v[1] : v[2];
}

template < typename T, typename A, int OP >
__global__ void __launch_bounds__( 256 ) k_cell_acc( int n, int nC, int nrows, const int2* __restrict__ rows, int nipts,
                                                      const ushort4* __restrict__ ipts, const int64_t* __restrict__ cell_off,
                                                      const uint8_t* __restrict__ cell_bc, uint32_t flag, AccVecs< T, A > vec,
                                                      const A* __restrict__ invd, A a0, A a1 )
{
   const A* __restrict__ acc = component( vec.acc, blockIdx.y );
   const T* src = component( vec.src, blockIdx.y );
   const T* v1  = component( vec.v1, blockIdx.y );
   T*       v2  = component( vec.v2, blockIdx.y );
   T*       dst = component( vec.dst, blockIdx.y );
   auto point = [&]( int64_t i ) {
      A       second;
      const A val = epilogue_value< T, A, OP >( i, acc[i], invd ? invd[i] : A( 1 ), src, v1, v2, a0, a1, &second );
      if constexpr ( OP == OP_CHEBL ) st_any( v2 + i, val );
      else if constexpr ( OP == OP_APPLY_ADD ) st_any( dst + i, A( ld_any( dst + i ) ) + val );
      else
      {
         st_any( dst + i, val );
         if constexpr ( OP == OP_CHEBI ) st_any( v2 + i, second );
      }
   };
   if ( n <= kFlatMaxN )
   {
      const int64_t g = int64_t( blockIdx.x ) * 256 + threadIdx.x;
      if ( g >= int64_t( nC ) * nipts ) return;
      const int c = g < 0x7fffffff ? int( unsigned( g ) / unsigned( nipts ) ) : int( g / nipts );
      if ( !( cell_bc[c] & flag ) ) return;
      const ushort4 p = ipts[int( g - int64_t( c ) * nipts )];
      point( cell_off[c] + cidx( n, p.x, p.y, p.z ) );
      return;
   }
   const int64_t w = int64_t( blockIdx.x ) * 8 + ( threadIdx.x >> 5 );
   if ( w >= int64_t( nC ) * nrows ) return;
   const int c = int( unsigned( w ) / unsigned( nrows ) );
   if ( !( cell_bc[c] & flag ) ) return;
   const int2    yz   = rows[int( w - int64_t( c ) * nrows )];
   const int64_t base = cell_off[c] + cidx( n, 0, yz.x, yz.y );
   for ( int x = 1 + ( threadIdx.x & 31 ); x <= n - 1 - yz.x - yz.y; x += 32 ) point( base + x );
}

template < typename T, typename A, int OP >
static void launch_cell_acc( Context* ctx, Mesh* m, const P1Level& P, uint32_t flag, const AccVecs< T, A >& vec, int ncomp, const A* invd, A a0,
                             A a1 )
{
   const int     nC = m->topo.nC, nrows = int( P.rows.size() );
   const int64_t blocks = P.n <= kFlatMaxN ? ( int64_t( nC ) * P.nipts + 255 ) / 256 : ( int64_t( nC ) * nrows + 7 ) / 8;
   if ( blocks == 0 ) return;
   k_cell_acc< T, A, OP ><<< dim3( unsigned( blocks ), ncomp ), 256, 0, ctx->stream >>>( P.n, nC, nrows, P.d_rows, P.nipts,
                                                                                        reinterpret_cast< const ushort4* >( P.d_ipts ),
                                                                                        P.d_off + P.nB, P.d_bc + P.nB, flag, vec, invd, a0, a1 );
   ++ctx->launches;
}

// cell-array slot of the copy of task tk's point in incidence I
__device__ __forceinline__ int64_t inc_slot( int n, const int4& tk, const Incidence& I, const int64_t* __restrict__ cell_off )
{
   const int x = n * I.o[0] + tk.y * I.e1[0] + tk.z * I.e2[0];
   const int y = n * I.o[1] + tk.y * I.e1[1] + tk.z * I.e2[1];
   const int z = n * I.o[2] + tk.y * I.e1[2] + tk.z * I.e2[2];
   return __ldg( cell_off + I.cell ) + cidx( n, x, y, z );
}

// owner and copies take val; the incidences are read four at a time ahead of their stores, so a
// vertex with many cells does not wait on one incidence read per copy
template < typename T, typename A >
__device__ __forceinline__ void wt_store( int n, const int4& tk, int64_t owner, const int* __restrict__ inc_begin,
                                          const Incidence* __restrict__ inc, const int64_t* __restrict__ cell_off, T* vec, A val )
{
   st_any( vec + owner, val );
   const int q1 = __ldg( inc_begin + tk.x + 1 );
   for ( int q = __ldg( inc_begin + tk.x ); q < q1; q += 4 )
   {
      int64_t sl[4];
#pragma unroll
      for ( int u = 0; u < 4; ++u ) sl[u] = q + u < q1 ? inc_slot( n, tk, inc[q + u], cell_off ) : -1;
#pragma unroll
      for ( int u = 0; u < 4; ++u )
         if ( sl[u] >= 0 ) st_any( vec + sl[u], val );
   }
}

// sum over the incidences q0..q1-1 of f(incidence), in incidence order, four incidences in flight
template < typename A, int U = 4, typename F >
__device__ __forceinline__ A inc_sum( int q0, int q1, const Incidence* __restrict__ inc, F f )
{
   A s = A( 0 );
   for ( int q = q0; q < q1; q += U )
   {
      A v[U];
#pragma unroll
      for ( int u = 0; u < U; ++u ) v[u] = q + u < q1 ? f( inc[q + u] ) : A( 0 );
#pragma unroll
      for ( int u = 0; u < U; ++u )
         if ( q + u < q1 ) s += v[u];
   }
   return s;
}

// Owners of face/edge/vertex DoFs: sum of the cell copies, epilogue, write-through.  G lanes per task
// (G = 1 on fine levels, where face points with two cells dominate; G = 8 on the coarsest levels,
// where a macro-vertex has 20-30 cells): the lanes of a task take every G-th incidence and combine
// their partial sums by a butterfly, which leaves the same bits in every lane of the group.
template < typename T, typename A, int OP, int G >
__global__ void __launch_bounds__( 256 ) k_bnd_acc( int n, int ntasks, const int4* __restrict__ tasks, const int64_t* __restrict__ off,
                                                     const int64_t* __restrict__ cell_off, const int8_t* __restrict__ bkind,
                                                     const uint8_t* __restrict__ bc, const int* __restrict__ inc_begin,
                                                     const Incidence* __restrict__ inc, uint32_t flag, int copy_unflagged,
                                                     AccVecs< T, A > vec, const A* __restrict__ invd, A* invd_out, A a0, A a1 )
{
   const A* __restrict__ acc = component( vec.acc, blockIdx.y );
   const T* src = component( vec.src, blockIdx.y );
   const T* v1  = component( vec.v1, blockIdx.y );
   T*       v2  = component( vec.v2, blockIdx.y );
   T*       dst = component( vec.dst, blockIdx.y );
   static_assert( G == 1 || G == 2 || G == 4 || G == 8 || G == 16 || G == 32, "G divides the warp" );
   const int gt = blockIdx.x * blockDim.x + threadIdx.x;
   const int t  = gt / G, sub = gt % G;
   if ( t >= ntasks ) return;  // a group's lanes share t: whole groups leave
   const int4    tk    = tasks[t];
   const int     b     = tk.x;
   const int     k     = bkind[b];
   const int64_t owner = off[b] + ( k == 0 ? 0 : ( k == 1 ? int64_t( tk.y ) : fidx( n, tk.y, tk.z ) ) );
   const int     q0 = __ldg( inc_begin + b ), q1 = __ldg( inc_begin + b + 1 );
   const unsigned gmask = G == 32 ? 0xffffffffu : ( ( 1u << G ) - 1u ) << ( ( threadIdx.x & 31 ) & ~( G - 1 ) );
   // this lane's share of the write-through (G = 1: the owner and every copy)
   auto store = [&]( T* vec, A val ) {
      if constexpr ( G == 1 ) wt_store< T, A >( n, tk, owner, inc_begin, inc, cell_off, vec, val );
      else
      {
         if ( sub == 0 ) st_any( vec + owner, val );
         for ( int q = q0 + sub; q < q1; q += G ) st_any( vec + inc_slot( n, tk, inc[q], cell_off ), val );
      }
   };
   if ( !( bc[b] & flag ) )
   {
      if ( !copy_unflagged ) return;
      if constexpr ( OP == OP_JAC || OP == OP_CHEB0 ) store( dst, A( ld_any( src + owner ) ) );
      else if constexpr ( OP == OP_CHEBI ) store( dst, A( ld_any( v2 + owner ) ) );
      return;
   }
   A s;
   if constexpr ( G == 1 )
      s = inc_sum< A >( q0, q1, inc, [&]( const Incidence& I ) { return acc[inc_slot( n, tk, I, cell_off )]; } );
   else
   {
      s = A( 0 );
      for ( int q = q0 + sub; q < q1; q += G ) s += acc[inc_slot( n, tk, inc[q], cell_off )];
#pragma unroll
      for ( int o = G / 2; o > 0; o >>= 1 ) s += __shfl_xor_sync( gmask, s, o, G );
   }
   if ( invd_out )  // diagonal setup: store 1/diag at the owner
   {
      if ( sub == 0 ) invd_out[owner] = A( 1 ) / s;
      return;
   }
   A       second;
   A       val = epilogue_value< T, A, OP >( owner, s, invd ? invd[owner] : A( 1 ), src, v1, v2, a0, a1, &second );
   if constexpr ( OP == OP_APPLY_ADD ) val = A( ld_any( dst + owner ) ) + val;
   // every lane of the group has read the owner's values before any lane stores
   if constexpr ( G > 1 ) __syncwarp( gmask );
   if constexpr ( OP == OP_CHEBL || OP == OP_APPLY_ADD ) store( OP == OP_CHEBL ? v2 : dst, val );
   else
   {
      store( dst, val );
      if constexpr ( OP == OP_CHEBI ) store( v2, second );
   }
}

// launch of the owner combine over the level's tasks, lanes per task by level size
template < typename T, typename A, int OP >
static void launch_bnd_acc( Context* ctx, cudaStream_t st, const P1Level& P, uint32_t flag, int copy_unflagged, const AccVecs< T, A >& vec,
                            int ncomp, const A* invd, A* invd_out, A a0, A a1 )
{
   const int nt = int( P.tasks.size() );
   if ( nt <= 0 ) return;
   if ( P.n <= 4 )
      k_bnd_acc< T, A, OP, 8 ><<< dim3( ( 8 * nt + 255 ) / 256, ncomp ), 256, 0, st >>>( P.n, nt, P.d_tasks, P.d_off, P.d_off + P.nB,
                                                                                        P.d_bkind, P.d_bc, P.d_inc_begin, P.d_inc, flag,
                                                                                        copy_unflagged, vec, invd, invd_out, a0, a1 );
   else
      k_bnd_acc< T, A, OP, 1 ><<< dim3( ( nt + 255 ) / 256, ncomp ), 256, 0, st >>>( P.n, nt, P.d_tasks, P.d_off, P.d_off + P.nB, P.d_bkind,
                                                                                    P.d_bc, P.d_inc_begin, P.d_inc, flag, copy_unflagged, vec,
                                                                                    invd, invd_out, a0, a1 );
   ++ctx->launches;
}

template < typename T, typename A >
static AccVecs< T, A > acc_vecs( const A* acc, const StencilArgs& a )
{
   AccVecs< T, A > v{};
   v.acc[0] = acc;
   v.src[0] = (const T*) a.src;
   v.v1[0]  = (const T*) a.v1;
   v.v2[0]  = (T*) a.v2;
   v.dst[0] = (T*) a.dst;
   return v;
}

// ---------------------------------------------------------------------------------------------
// Assembled stencils (P1 operators with stored matrices): A src at cell-local (x, y, z) of a cell is
// sum_d S_d(slot) src(x + dir_d), S_d the sum of the element-matrix entries of the cell's micro-cells
// that couple the point with its neighbour in direction d (the same sum the elementwise apply forms,
// P1ElementwiseOperator.cpp:169-260, taken once at setup instead of every apply).  The matrices are
// symmetric, so only the centre and one direction of each opposite pair are kept, eight values per slot
// (kVarDirs lists opposite directions next to each other: 2k - 1 is minus 2k); the other seven are the
// neighbours' values for the direction back.
//
// One thread per cell-array slot, so warps are full whatever the length of the rows (a warp per row left
// two thirds of its lanes idle at 32 points per edge).  Bound by the weights: 64 bytes per slot from
// memory in FP64, the other 56 from cache.  Inner points finish here, points on the cell's boundary leave
// their partial sums in acc for the owners (a gather of their weights by the owners took as long as the
// whole interior).  V(3,3) Chebyshev(3) cycle on a shell of 240 cells, levels 0-5, FP64: 8.59 ms with a warp
// per row, 15 stored weights and gathering owners, 3.62 ms so.
// ---------------------------------------------------------------------------------------------
template < int D, typename T, typename A >
__device__ __forceinline__ void var_term( const A* S, int64_t ssize, const T* src, int n, int x, int y, int z, bool inner, A ( &s )[3] )
{
   constexpr int dx = StencilDir< D >::x, dy = StencilDir< D >::y, dz = StencilDir< D >::z;
   if ( !inner && ( x + dx < 0 || y + dy < 0 || z + dz < 0 || x + y + z + ( dx + dy + dz ) > n ) ) return;
   const int o = row_shift< dy, dz >( n, y, z ) + dx;
   const A   w = ( D & 1 ) ? __ldg( S + ( ( D + 1 ) / 2 ) * ssize + o ) : __ldg( S + ( D / 2 ) * ssize );
   s[D % 3] += w * A( ld_any( src + o ) );
}

template < typename T, typename A, int... D >
__device__ __forceinline__ A var_sum( const A* S, int64_t ssize, const T* src, int n, int x, int y, int z, bool inner,
                                      std::integer_sequence< int, D... > )
{
   A s[3] = { A( 0 ), A( 0 ), A( 0 ) };
   ( var_term< D, T, A >( S, ssize, src, n, x, y, z, inner, s ), ... );
   return ( s[0] + s[1] ) + s[2];
}

template < typename T, typename A, int OP >
__global__ void __launch_bounds__( 256 ) k_var_sweep( int n, int nC, int np, int cell_stride, const ushort4* __restrict__ pts,
                                                       const int64_t* __restrict__ cell_off, const uint8_t* __restrict__ cell_bc, uint32_t flag,
                                                       const A* __restrict__ S, int64_t ssize, const A* __restrict__ invd,
                                                       A* __restrict__ acc, const T* src, const T* v1, T* v2, T* dst, A a0, A a1 )
{
   // threads over the slots of all macro-cells in storage order
   const int64_t g = int64_t( blockIdx.x ) * 256 + threadIdx.x;
   if ( g >= int64_t( nC ) * cell_stride ) return;
   const int c = g < 0x7fffffff ? int( unsigned( g ) / unsigned( cell_stride ) ) : int( g / cell_stride );
   const int k = int( g - int64_t( c ) * cell_stride );
   if ( k >= np ) return;  // padding
   const ushort4 pt    = pts[k];
   const int     x = pt.x, y = pt.y, z = pt.z;
   const bool    inner = x > 0 && y > 0 && z > 0 && x + y + z < n;
   if ( inner && !( cell_bc[c] & flag ) ) return;
   const int64_t i = cell_off[c] + k;
   const A       s = var_sum< T, A >( S + i, ssize, src + i, n, x, y, z, inner, std::make_integer_sequence< int, 15 >() );
   if ( !inner )
   {
      acc[i] = s;
      return;
   }
   A       second;
   const A val = epilogue_value< T, A, OP >( i, s, invd[i], src, v1, v2, a0, a1, &second );
   if constexpr ( OP == OP_CHEBL ) st_any( v2 + i, val );
   else if constexpr ( OP == OP_APPLY_ADD ) st_any( dst + i, A( ld_any( dst + i ) ) + val );
   else
   {
      st_any( dst + i, val );
      if constexpr ( OP == OP_CHEBI ) st_any( v2 + i, second );
   }
}

// Stored stencils on levels whose tasks are edges and vertices alone: P1 levels 0 and 1, P2 level 0 (two
// storage points per edge).  A sweep would only fill partial sums, and its launch and the wait for it are most of
// the time there (shell of 240 cells: P1 apply on level 0, all vertices on the boundary, 12.6 us with a sweep and
// the owners' combine and 2.9 us so, P2 level 0 19.3 and 8.8), so the owners gather from their cells at once, eight
// threads each.  part( I ): the sum of incidence I's cell.
template < typename T, typename A, int OP, typename F >
__device__ __forceinline__ void low_owner( const LevelView& v, const BndSegments& seg, uint32_t flag, int copy_unflagged, const A* invd,
                                           const T* src, const T* v1, T* v2, T* dst, A a0, A a1, F part )
{
   LowRec    low;
   FaceRec   none;
   int       sub;
   if ( bnd_thread< 1 >( v, v.frec, seg, int( blockIdx.x * blockDim.x + threadIdx.x ), low, sub, none ) != BND_LOW ) return;
   constexpr bool CARRIES = OP == OP_JAC || OP == OP_CHEB0 || OP == OP_CHEBI;
   const bool     flagged = ( low.bc & flag ) != 0;
   if ( !flagged && !( CARRIES && copy_unflagged ) ) low.count = 0;
   A val = A( 0 ), second = A( 0 ), s = A( 0 );
   if ( flagged )
      for ( int q = sub; q < low.count; q += 8 ) s += part( v.irec[low.begin + q] );
#pragma unroll
   for ( int m = 4; m > 0; m >>= 1 ) s += __shfl_xor_sync( 0xffffffffu, s, m, 8 );
   if ( low.count > 0 )
   {
      if ( flagged ) val = owner_value< T, A >( OP, low.owner, s, invd[low.owner], src, v1, v2, dst, a0, a1, second );
      else if constexpr ( OP == OP_JAC || OP == OP_CHEB0 ) val = A( ldv( src + low.owner ) );
      else if constexpr ( OP == OP_CHEBI ) val = A( ldc( v2 + low.owner ) );
   }
   __syncwarp();  // every thread of a task has read the owner before any writes it
   put_low( v, low, sub, OP == OP_CHEBL ? v2 : dst, val );
   if constexpr ( OP == OP_CHEBI )
      if ( flagged ) put_low( v, low, sub, v2, second );
}

template < typename T, typename A, int OP >
__global__ void __launch_bounds__( 256 ) k_var_low( LevelView v, BndSegments seg, uint32_t flag, int copy_unflagged, const A* __restrict__ S,
                                                     int64_t ssize, const A* __restrict__ invd, const T* src, const T* v1, T* v2, T* dst,
                                                     A a0, A a1 )
{
   low_owner< T, A, OP >( v, seg, flag, copy_unflagged, invd, src, v1, v2, dst, a0, a1, [&]( const IncRec& I ) {
      return var_sum< T, A >( S + I.slot, ssize, src + I.slot, v.n, I.x, I.y, I.z, false, std::make_integer_sequence< int, 15 >() );
   } );
}

// P2 level 0: a macro-cell is one micro-cell, and a node's row its ten nodes (component: blockIdx.y)
template < typename T, typename A, int OP >
__global__ void __launch_bounds__( 256 ) k_p2_stored_low( LevelView v, BndSegments seg, P2StoredView sv, uint32_t flag, int copy_unflagged,
                                                           const A* __restrict__ S, const A* __restrict__ invd, AccVecs< T, A > vec, A a0,
                                                           A a1 )
{
   const T* src = component( vec.src, blockIdx.y );
   low_owner< T, A, OP >( v, seg, flag, copy_unflagged, invd, src, component( vec.v1, blockIdx.y ), component( vec.v2, blockIdx.y ),
                          component( vec.dst, blockIdx.y ), a0, a1, [&]( const IncRec& I ) {
                             int64_t       skip;
                             const int64_t w = p2_weight_at( sv, I.cell, I.x, I.y, I.z, skip );
                             const int     i = c_p2_node0[I.x + 3 * I.y + 9 * I.z];
                             const int64_t c = v.cell_off[I.cell];
                             A             sum = A( 0 );
#pragma unroll
                             for ( int j = 0; j < 10; ++j )
                             {
                                const int l = c_p2_loc[0][j];
                                sum += __ldg( S + w + c_p2s_ent[10 * i + j] * skip ) * A( ldv( src + c + cidx( 2, l % 3, ( l / 3 ) % 3, l / 9 ) ) );
                             }
                             return sum;
                          } );
}

template < typename A >
__global__ void k_cell_invert( int n, int nrows, const int2* __restrict__ rows, const int64_t* __restrict__ cell_off, const A* acc,
                               A* invd )
{
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const int r    = blockIdx.x * 8 + warp;
   const int c    = blockIdx.y;
   if ( r >= nrows ) return;
   const int2    yz   = rows[r];
   const int64_t base = cell_off[c] + cidx( n, 0, yz.x, yz.y );
   for ( int x = 1 + lane; x <= n - 1 - yz.x - yz.y; x += 32 ) invd[base + x] = A( 1 ) / acc[base + x];
}

// ---------------------------------------------------------------------------------------------
// Stokes coupling blocks (P2P1ElementwiseBlendingStokesOperator, P2P1ElementwiseBlendingStokesOperator.hpp:
// 113-116): div = P2ToP1ElementwiseBlendingDiv{x,y,z} (forms p2_to_p1_div_{0,1,2}_blending_q2) maps a
// P2 velocity of level l to a P1 pressure of level l, divT (p1_to_p2_divt_{0,1,2}_blending_q2) is its
// transpose.  Element matrix of component k: B_k[i][j] = -int psi_i d(phi_j)/dx_k over the blended
// micro-cell, psi P1 and phi P2, with the 4-point degree-2 rule (a = (5 - sqrt 5)/20,
// b = (5 + 3 sqrt 5)/20, weights 1/24).  Applied matrix-free: div forms the divergence of the local
// velocity at each point; divT pairs the local pressure with every basis gradient.  The P1 nodes are
// the micro-cell's vertices on level l, the P2 nodes the ten nodes on storage level l+1; anchors of
// one parity class share neither, so the passes are race-free.
// ---------------------------------------------------------------------------------------------
__constant__ double c_q2_bary[4][4];

void ensure_stokes_constants()
{
   static PerDeviceOnce once;
   once.run( [] {
      const double a = ( 5.0 - std::sqrt( 5.0 ) ) / 20.0, b = ( 5.0 + 3.0 * std::sqrt( 5.0 ) ) / 20.0;
      const double c = 1.0 - 3.0 * a, e = 1.0 - 2.0 * a - b;
      const double bary[4][4] = { { c, a, a, a }, { e, b, a, a }, { e, a, b, a }, { e, a, a, b } };
      check_cuda( cudaMemcpyToSymbol( c_q2_bary, bary, sizeof( bary ) ), "Stokes constants (points)" );
   } );
}

// inverse of the blended Jacobian M = DF J at reference point xi and |det M|
// (Fq, when given, receives the blended point)
template < typename A >
__device__ __forceinline__ void mapped_point( const CellGeom& g, const A X0[3], const A J[3][3], const double* xi, A Mi[3][3], A& adet,
                                              A* Fq = nullptr )
{
   A Xq[3];
   for ( int r = 0; r < 3; ++r ) Xq[r] = X0[r] + J[r][0] * A( xi[0] ) + J[r][1] * A( xi[1] ) + J[r][2] * A( xi[2] );
   A M[3][3];
   if ( g.blend == 1 )
   {
      A DF[3][3], Fl[3];
      shell_map( g, Xq, Fl, DF );
      for ( int r = 0; r < 3; ++r )
         for ( int c = 0; c < 3; ++c ) M[r][c] = DF[r][0] * J[0][c] + DF[r][1] * J[1][c] + DF[r][2] * J[2][c];
      if ( Fq )
         for ( int r = 0; r < 3; ++r ) Fq[r] = Fl[r];
   }
   else
   {
      for ( int r = 0; r < 3; ++r )
         for ( int c = 0; c < 3; ++c ) M[r][c] = J[r][c];
      if ( Fq )
         for ( int r = 0; r < 3; ++r ) Fq[r] = Xq[r];
   }
   const A c00 = M[1][1] * M[2][2] - M[1][2] * M[2][1];
   const A c01 = M[1][2] * M[2][0] - M[1][0] * M[2][2];
   const A c02 = M[1][0] * M[2][1] - M[1][1] * M[2][0];
   const A det = M[0][0] * c00 + M[0][1] * c01 + M[0][2] * c02;
   const A id  = A( 1 ) / det;
   Mi[0][0]    = c00 * id;
   Mi[1][0]    = c01 * id;
   Mi[2][0]    = c02 * id;
   Mi[0][1]    = ( M[0][2] * M[2][1] - M[0][1] * M[2][2] ) * id;
   Mi[1][1]    = ( M[0][0] * M[2][2] - M[0][2] * M[2][0] ) * id;
   Mi[2][1]    = ( M[0][1] * M[2][0] - M[0][0] * M[2][1] ) * id;
   Mi[0][2]    = ( M[0][1] * M[1][2] - M[0][2] * M[1][1] ) * id;
   Mi[1][2]    = ( M[0][2] * M[1][0] - M[0][0] * M[1][2] ) * id;
   Mi[2][2]    = ( M[0][0] * M[1][1] - M[0][1] * M[1][0] ) * id;
   adet        = fabs( det );
}

// The coupled passes compute a micro-cell in FP64 for every value type and only the coefficient in the
// accumulation type: their results are sums of terms of either sign (the divergence, the negative weight of
// the five-point rule), which in FP32 lost up to 1.8 times as much as evaluating every point by itself.

// B u of one micro-cell: the pressure values of its vertices from the velocity's node values
__device__ __forceinline__ void div_micro( const MicroCell< double >& mc, bool blend, const double ( &ul )[3][10], double ( &yl )[4] )
{
   const double wj = -( 1.0 / 24.0 ) * mc.adet;
   double       G[3][4][3];
#pragma unroll
   for ( int k = 0; k < 3; ++k ) p2_vertex_gradients( ul[k], mc.Ji, G[k] );
   for ( int i = 0; i < 4; ++i ) yl[i] = 0;
#pragma unroll 1
   for ( int q = 0; q < 4; ++q )
   {
      const double lam[4] = { c_q2_bary[q][0], c_q2_bary[q][1], c_q2_bary[q][2], c_q2_bary[q][3] };
      // velocity gradient B with respect to X; div = (tr B - g^T B X / m) / s and |det DF| = s^2 |m|
      double B[3][3];
#pragma unroll
      for ( int k = 0; k < 3; ++k )
#pragma unroll
         for ( int d = 0; d < 3; ++d ) B[k][d] = lam[0] * G[k][0][d] + lam[1] * G[k][1][d] + lam[2] * G[k][2][d] + lam[3] * G[k][3][d];
      double f = B[0][0] + B[1][1] + B[2][2];
      if ( blend )
      {
         ShellPoint< double > p;
         cell_point( mc, lam[1], lam[2], lam[3], p );
         shell_point( mc, lam[1], lam[2], lam[3], p );
         double gbx = 0;
#pragma unroll
         for ( int k = 0; k < 3; ++k ) gbx += p.g[k] * ( B[k][0] * p.X[0] + B[k][1] * p.X[1] + B[k][2] * p.X[2] );
         f = ( f - gbx * p.im ) * ( p.s * fabs( p.m ) );
      }
      f *= wj;
#pragma unroll
      for ( int i = 0; i < 4; ++i ) yl[i] += f * lam[i];
   }
}

// B^T p of one micro-cell: the velocity's node values from the vertices' pressures
__device__ __forceinline__ void divt_micro( const MicroCell< double >& mc, bool blend, const double ( &pl )[4], double ( &yl )[3][10] )
{
   const double wj = -( 1.0 / 24.0 ) * mc.adet;
   double       H[3][4][3];
#pragma unroll
   for ( int k = 0; k < 3; ++k )
#pragma unroll
      for ( int v = 0; v < 4; ++v ) H[k][v][0] = H[k][v][1] = H[k][v][2] = 0;
#pragma unroll 1
   for ( int q = 0; q < 4; ++q )
   {
      const double lam[4] = { c_q2_bary[q][0], c_q2_bary[q][1], c_q2_bary[q][2], c_q2_bary[q][3] };
      double       f      = wj * ( pl[0] * lam[0] + pl[1] * lam[1] + pl[2] * lam[2] + pl[3] * lam[3] );
      // component k pairs with DF^-1 e_k |det DF| = s |m| (e_k - X g_k / m)
      double E[3][3] = { { 1, 0, 0 }, { 0, 1, 0 }, { 0, 0, 1 } };
      if ( blend )
      {
         ShellPoint< double > p;
         cell_point( mc, lam[1], lam[2], lam[3], p );
         shell_point( mc, lam[1], lam[2], lam[3], p );
#pragma unroll
         for ( int k = 0; k < 3; ++k )
         {
            const double gk = p.g[k] * p.im;
#pragma unroll
            for ( int d = 0; d < 3; ++d ) E[k][d] -= p.X[d] * gk;
         }
         f *= p.s * fabs( p.m );
      }
#pragma unroll
      for ( int v = 0; v < 4; ++v )
      {
         const double fl = f * lam[v];
#pragma unroll
         for ( int k = 0; k < 3; ++k )
#pragma unroll
            for ( int d = 0; d < 3; ++d ) H[k][v][d] += fl * E[k][d];
      }
   }
#pragma unroll
   for ( int k = 0; k < 3; ++k ) p2_pair_gradients( H[k], mc.Ji, yl[k] );
}

// the full viscous block of one micro-cell on its three components' node values (the coefficient in A)
template < typename A >
__device__ __forceinline__ void visc_micro( const MicroCell< double >& mc, bool blend, const Coefficient& kc, const double ( &ul )[3][10],
                                            double ( &yl )[3][10] )
{
   double G[3][4][3], H[3][4][3];
#pragma unroll
   for ( int k = 0; k < 3; ++k )
   {
      p2_vertex_gradients( ul[k], mc.Ji, G[k] );
#pragma unroll
      for ( int v = 0; v < 4; ++v ) H[k][v][0] = H[k][v][1] = H[k][v][2] = 0;
   }
#pragma unroll 1
   for ( int q = 0; q < 5; ++q )
   {
      const double l1 = c_yu5_pts[q][0], l2 = c_yu5_pts[q][1], l3 = c_yu5_pts[q][2], l0 = 1 - l1 - l2 - l3;
      double       D[3][3];  // velocity gradient, d u_k / d x_d
#pragma unroll
      for ( int k = 0; k < 3; ++k )
#pragma unroll
         for ( int d = 0; d < 3; ++d ) D[k][d] = l0 * G[k][0][d] + l1 * G[k][1][d] + l2 * G[k][2][d] + l3 * G[k][3][d];
      ShellPoint< double > p;
      cell_point( mc, l1, l2, l3, p );
      double f = c_yu5_w[q] * mc.adet;
      A      F[3] = { A( p.X[0] ), A( p.X[1] ), A( p.X[2] ) }, rad = A( -1 );
      if ( blend )
      {
         // |det DF| = s^2 |m| takes the two factors 1/s of DF^-T and DF^-1
         shell_point( mc, l1, l2, l3, p );
#pragma unroll
         for ( int k = 0; k < 3; ++k )
         {
            const double xb = ( p.X[0] * D[k][0] + p.X[1] * D[k][1] + p.X[2] * D[k][2] ) * p.im;
#pragma unroll
            for ( int d = 0; d < 3; ++d ) D[k][d] -= p.g[d] * xb;
            F[k] = A( p.X[k] * p.s );
         }
         f *= fabs( p.m );
         rad = A( p.R );
      }
      f *= double( coeff_eval( kc, F, rad ) );
      const double tr3     = ( 2.0 / 3.0 ) * ( D[0][0] + D[1][1] + D[2][2] );
      double       S[3][3] = { { D[0][0] + D[0][0] - tr3, D[0][1] + D[1][0], D[0][2] + D[2][0] },
                               { D[0][1] + D[1][0], D[1][1] + D[1][1] - tr3, D[1][2] + D[2][1] },
                               { D[0][2] + D[2][0], D[1][2] + D[2][1], D[2][2] + D[2][2] - tr3 } };
#pragma unroll
      for ( int k = 0; k < 3; ++k )
      {
         if ( blend )
         {
            const double gs = ( p.g[0] * S[k][0] + p.g[1] * S[k][1] + p.g[2] * S[k][2] ) * p.im;
#pragma unroll
            for ( int d = 0; d < 3; ++d ) S[k][d] -= p.X[d] * gs;
         }
#pragma unroll
         for ( int d = 0; d < 3; ++d )
         {
            const double h = f * S[k][d];
            H[k][0][d] += l0 * h;
            H[k][1][d] += l1 * h;
            H[k][2][d] += l2 * h;
            H[k][3][d] += l3 * h;
         }
      }
   }
#pragma unroll
   for ( int k = 0; k < 3; ++k ) p2_pair_gradients( H[k], mc.Ji, yl[k] );
}

// One parity pass of a coupled operator, a thread per micro-cell: warp w takes type w of the block's 32
// anchors.  The six micro-cells of an anchor share nodes, so their results meet in shared memory and are
// added to the accumulators once per node, in a fixed order.  A thread per anchor walked its six
// micro-cells one after the other, 20 to 40 us a pass on levels whose classes have a few thousand anchors.
// Full viscous apply, shell of 480 cells, level 3: 399 -> 341 us; of 240 cells, level 2: 630 us with the
// element loops of 10 basis gradients, 187 us so; 960 cells, level 4: 4.71 -> 2.69 ms.  At 168 registers two
// blocks fit an SM.
enum { CPL_VISCOUS = 0, CPL_DIVT, CPL_DIV };
template < typename T, typename A >
struct CoupledArgs {
   const T* u[3];
   const T* p;
   A*       acc[3];  // velocity components, or the pressure in acc[0]
};
constexpr int kCoupledThreads = 192;
template < typename T, typename A, int OPER >
__global__ void __launch_bounds__( kCoupledThreads, 2 )
    k_coupled_pass( int ne, int nC, int nanch, const int* __restrict__ anch, const int64_t* __restrict__ off_p, const int64_t* __restrict__ off_u,
                    const CellGeom* __restrict__ geom, Coefficient kc, CoupledArgs< T, A > v, int64_t size_p, int64_t size_u, int* err )
{
   constexpr int NC = OPER == CPL_DIV ? 1 : 3, NN = OPER == CPL_DIV ? 4 : 10;  // result components, nodes per micro-cell
   __shared__ A  ys[NC][6 * NN][32];
   const int     ty = threadIdx.x >> 5, lane = threadIdx.x & 31, ns = 2 * ne;
   const int64_t t    = int64_t( blockIdx.x ) * 32 + lane;
   bool          live = t < int64_t( nC ) * nanch;
   const int64_t tt   = live ? t : 0;
   const int     c    = tt < 0x7fffffff ? int( unsigned( tt ) / unsigned( nanch ) ) : int( tt / nanch );
   const int     a    = anch[int( tt - int64_t( c ) * nanch )];
   const int     x = a & 1023, y = ( a >> 10 ) & 1023, z = a >> 20, room = ns - 2 * ( x + y + z );
   const int64_t bu = off_u[c], bp = off_p ? off_p[c] : 0;
   {
      // self-check: every node of the windows inside the level's vectors
      const int64_t lu = bu + window_last( ns, 2 * x, 2 * y, 2 * z, 2, room ), lp = bp + window_last( ne, x, y, z, 1, room / 2 );
      if ( live && ( room < 2 || bu < 0 || lu >= size_u || ( off_p && ( bp < 0 || lp >= size_p ) ) ) )
      {
         atomicExch( err, 2 );
         live = false;
      }
   }
   auto at_u = [&]( int l ) { return bu + cidx( ns, 2 * x + l % 3, 2 * y + ( l / 3 ) % 3, 2 * z + l / 9 ); };
   auto at_p = [&]( int l ) { return bp + cidx( ne, x + ( l & 1 ), y + ( ( l >> 1 ) & 1 ), z + ( l >> 2 ) ); };
   // vertex i of the type: its number x + 2 y + 4 z among the anchor's eight
   auto vert = [&]( int i ) {
      const int l = c_p2_loc[ty][i];
      return ( l % 3 ) / 2 + ( l / 3 ) % 3 / 2 * 2 + l / 9 / 2 * 4;
   };
   if ( live && x + y + z <= ne - 1 - c_mc_shift[ty] )
   {
      const CellGeom&     g     = geom[c];
      const bool          blend = g.blend == 1;
      MicroCell< double > mc;
      micro_cell( g, ne, ty, x, y, z, mc );
      double yl[NC][NN];
      if constexpr ( OPER == CPL_DIVT )
      {
         double pl[4];
#pragma unroll
         for ( int i = 0; i < 4; ++i ) pl[i] = double( ld_any( v.p + at_p( vert( i ) ) ) );
         divt_micro( mc, blend, pl, yl );
      }
      else
      {
         double ul[3][10];
#pragma unroll
         for ( int i = 0; i < 10; ++i )
         {
            const int64_t at = at_u( c_p2_loc[ty][i] );
#pragma unroll
            for ( int k = 0; k < 3; ++k ) ul[k][i] = double( ld_any( v.u[k] + at ) );
         }
         if constexpr ( OPER == CPL_VISCOUS ) visc_micro< A >( mc, blend, kc, ul, yl );
         else div_micro( mc, blend, ul, yl[0] );
      }
#pragma unroll
      for ( int k = 0; k < NC; ++k )
#pragma unroll
         for ( int i = 0; i < NN; ++i ) ys[k][NN * ty + i][lane] = A( yl[k][i] );
   }
   else
#pragma unroll
      for ( int k = 0; k < NC; ++k )
#pragma unroll
         for ( int i = 0; i < NN; ++i ) ys[k][NN * ty + i][lane] = A( 0 );
   __syncthreads();
   if ( !live ) return;
   if constexpr ( OPER == CPL_DIV )
   {
      for ( int l = ty; l < 8; l += 6 )
      {
         const int dx = l & 1, dy = ( l >> 1 ) & 1, dz = l >> 2, w = 2 * dx + 6 * dy + 18 * dz;
         if ( 2 * ( dx + dy + dz ) > room ) continue;
         A s = A( 0 );
         for ( int k = c_p2_from0[w]; k < c_p2_from0[w + 1]; ++k )
            s += ys[0][4 * ( c_p2_from[k] / 10 ) + c_p2_from[k] % 10][lane];  // a vertex of the window is one of every micro-cell that has it
         v.acc[0][at_p( l )] += s;
      }
   }
   else
      for ( int l = ty; l < 27; l += 6 )
      {
         if ( l % 3 + ( l / 3 ) % 3 + l / 9 > room ) continue;
         A s[NC];
#pragma unroll
         for ( int j = 0; j < NC; ++j ) s[j] = A( 0 );
         for ( int k = c_p2_from0[l]; k < c_p2_from0[l + 1]; ++k )
#pragma unroll
            for ( int j = 0; j < NC; ++j ) s[j] += ys[j][c_p2_from[k]][lane];
         const int64_t at = at_u( l );
#pragma unroll
         for ( int j = 0; j < NC; ++j ) v.acc[j][at] += s[j];
      }
}

// ---------------------------------------------------------------------------------------------
// host launch
// ---------------------------------------------------------------------------------------------
template < typename A >
static A* acc_buffer( Operator* op, int L, int64_t size )
{
   ElemLevel& e   = op->el[L];
   const int  adt = sizeof( A ) == 8 ? F64 : F32;
   if ( e.d_acc && e.acc_dtype != adt && adt == F64 )
   {
      check_cuda( cudaFree( e.d_acc ), "cudaFree(acc)" );
      e.d_acc = nullptr;
   }
   if ( !e.d_acc )
   {
      check_cuda( cudaMalloc( &e.d_acc, size * sizeof( double ) ), "cudaMalloc(elementwise scratch)" );
      e.acc_dtype = F64;
   }
   return reinterpret_cast< A* >( e.d_acc );
}

// stencil direction of every vertex pair of every micro-cell type (vertex offsets as c_mc_off)
static void ensure_var_tables()
{
   static PerDeviceOnce once;
   once.run( [] {
      int off[6][4][3];
      for ( int t = 0; t < 6; ++t )
         for ( int i = 0; i < 4; ++i )
            for ( int d = 0; d < 3; ++d ) off[t][i][d] = micro_vertex( t, i, d );
      int8_t dir[6][4][4];
      for ( int t = 0; t < 6; ++t )
         for ( int i = 0; i < 4; ++i )
            for ( int j = 0; j < 4; ++j )
            {
               int found = -1;
               for ( int d = 0; d < 15; ++d )
                  if ( off[t][j][0] - off[t][i][0] == kVarDirs[d][0] && off[t][j][1] - off[t][i][1] == kVarDirs[d][1] &&
                       off[t][j][2] - off[t][i][2] == kVarDirs[d][2] )
                     found = d;
               if ( found < 0 ) throw std::runtime_error( "micro-cell edge outside the 15-point stencil" );
               dir[t][i][j] = int8_t( found );
            }
      check_cuda( cudaMemcpyToSymbol( c_mc_dir, dir, sizeof( dir ) ), "upload stencil directions" );
   } );
}

template < typename A >
static A* assembled_stencils( Operator* op, int L ) { return reinterpret_cast< A* >( op->el[L].d_S[sizeof( A ) == 8 ? 0 : 1] ); }

// micro-cells per macro-edge of the elements living on storage level L (P2 elements of level L-1
// have their nodes on storage level L)
static int element_n( const Operator* op, int L ) { return op->order == 2 ? ( 1 << ( L - 1 ) ) : ( 1 << L ); }

// micro-cell anchors (x, y, z), x + y + z <= n - 1, grouped by coordinate parity: the micro-cells of
// anchors of one parity class share no vertex (nor, for P2, any node), so a pass over one class
// updates its nodes without conflicts
static void ensure_rows( Operator* op, int L )
{
   ElemLevel& e = op->el[L];
   if ( e.d_anch ) return;
   const int          n = element_n( op, L );
   std::vector< int > anch;
   TableArrays        arrays;
   for ( int p = 0; p < 8; ++p )
   {
      e.aoff[p]    = int( anch.size() );
      const int px = p & 1, py = ( p >> 1 ) & 1, pz = p >> 2;
      // P2: by the number of micro-cells an anchor has (six; five next to the slanted face; one at it), so
      // that the threads of a warp visit the same micro-cell types.  P1: in storage order, whose warps touch fewer
      // sectors (level 4, FP32: 17 to 19 us a pass, 18 to 22 by kind).
      for ( int k = 0; k < 3; ++k )
      {
         int lo = k == 0 ? 0 : n - 3 + k, hi = n - 3 + k;
         if ( op->order == 1 ) lo = k == 0 ? 0 : n, hi = n - 1;
         const int before = int( anch.size() );
         for ( int z = pz; z <= n - 1; z += 2 )
            for ( int y = py; y + z <= n - 1; y += 2 )
               for ( int x = px; x + y + z <= n - 1; x += 2 )
                  if ( x + y + z >= lo && x + y + z <= hi ) anch.push_back( x | ( y << 10 ) | ( z << 20 ) );
         e.akind[p][k] = int( anch.size() ) - before;
      }
   }
   e.aoff[8] = int( anch.size() );
   int* d_anch = arrays.upload( anch.data(), anch.size(), "anchors" );
   arrays.keep();
   e.d_anch = d_anch;
}

// threads per block of a pass over na anchors per cell (grid: blocks x cells): whole warps, at most
// maxb, so that the small levels (a few anchors per cell) do not launch mostly idle blocks
static int pass_block( int na, int maxb ) { return std::min( maxb, ( na + 31 ) / 32 * 32 ); }

// (MODE 2 and 4: the stencils st, for P2 of the layout sv and st_size values, which a failure leaves unpublished;
// MODE 2: the cells first_cell .. first_cell + sv->nC - 1)
template < typename T, typename A, int MODE >
static void run_passes( Context* ctx, Mesh* m, Operator* op, int L, const T* src, A* acc, A* st = nullptr, const P2StoredView* sv = nullptr,
                        int64_t st_size = 0, int first_cell = 0 )
{
   P1Level&   P = m->level( L );
   ElemLevel& e = op->el[L];
   if ( MODE != 2 && MODE != 4 ) check_cuda( cudaMemsetAsync( acc, 0, P.size * sizeof( A ), ctx->stream ), "cudaMemset(acc)" );
   const int nC = MODE == 2 ? sv->nC : m->topo.nC;
   for ( int p = 0; p < 8; ++p )
   {
      const int na = e.aoff[p + 1] - e.aoff[p];
      if ( na <= 0 ) continue;
      const int bs = pass_block( na, op->order == 1 ? 128 : 256 );
      dim3      grid( ( na + bs - 1 ) / bs, nC );
      if ( op->order == 2 && MODE == 0 )
      {
         const int3 kinds  = make_int3( e.akind[p][0], e.akind[p][1], e.akind[p][2] );
         // anchors that the SMs with six blocks of k_p2_apply_pass each hold at once (56,832 on 148 SMs): below it
         // the split pass is faster (shell of 240 cells, level 3: 183 against 494 us an apply), above it slower
         // (2.69 against 2.27 ms on the shell named there)
         const bool split  = int64_t( na ) * nC < int64_t( ctx->sms ) * 6 * kP2ApplyThreads;
         const int  per    = split ? 32 : kP2ApplyThreads, per1 = split ? kP2SplitThreads : kP2ApplyThreads;
         auto       blocks = [&]( int k, int b ) { return int( ( int64_t( k ) * nC + b - 1 ) / b ); };
         const int3 bl     = make_int3( blocks( kinds.x, per ), blocks( kinds.y, per ), blocks( kinds.z, per1 ) );
         auto       launch = [&]( auto nodal, auto blend ) {
            constexpr bool NODAL = decltype( nodal )::value, BLEND = decltype( blend )::value;
            const double*  kn    = NODAL ? e.d_kn : nullptr;
            const int      pg    = bl.x + bl.y + bl.z;
            if ( split )
               k_p2_apply_split< T, A, NODAL, BLEND ><<< pg, kP2SplitThreads, 0, ctx->stream >>>( element_n( op, L ), nC, kinds, bl, e.d_anch + e.aoff[p],
                                                                                          P.d_off + P.nB, op->d_geom, op->coeff, src, acc,
                                                                                          P.size, ctx->d_error, kn );
            else
               k_p2_apply_pass< T, A, NODAL, BLEND ><<< pg, kP2ApplyThreads, 54 * kP2ApplyThreads * sizeof( A ), ctx->stream >>>(
                   element_n( op, L ), nC, kinds, bl, e.d_anch + e.aoff[p], P.d_off + P.nB, op->d_geom, op->coeff, src, acc, P.size,
                   ctx->d_error, kn );
         };
         if ( op->nodal_k && op->blending == 1 ) launch( std::true_type{}, std::true_type{} );
         else if ( op->nodal_k ) launch( std::true_type{}, std::false_type{} );
         else if ( op->blending == 1 ) launch( std::false_type{}, std::true_type{} );
         else launch( std::false_type{}, std::false_type{} );
      }
      else if ( op->order == 2 && ( MODE == 1 || MODE == 2 ) )
         k_p2_pass< A, MODE == 2 ? 2 : 1 ><<< grid, bs, 0, ctx->stream >>>( element_n( op, L ), first_cell, na, e.d_anch + e.aoff[p], P.d_off + P.nB,
                                                                            op->d_geom, op->coeff, acc, sv ? *sv : P2StoredView{}, st, st_size, P.size,
                                                                            ctx->d_error, op->nodal_k ? e.d_kn : nullptr );
      else if constexpr ( MODE != 2 )
         k_elem_pass< T, A, MODE ><<< grid, bs, 0, ctx->stream >>>( P.n, na, e.d_anch + e.aoff[p], P.d_off + P.nB, op->d_geom, op->coeff,
                                                                    src, acc, st, P.size, P.size, ctx->d_error );
      ++ctx->launches;
   }
   check_cuda( cudaGetLastError(), "elementwise pass launch" );
}

// A coefficient stored as a P2 function (the hyteg-operators P2ElementwiseDivKGrad operators take k
// as a P2Function interpolated at the nodes): its closed form at every cell-array node of storage
// level ns, at the node's blended position.  Block (z, cell), threads over the rows y of slice z.
__global__ void __launch_bounds__( 128 ) k_p2_nodal_coeff( int ns, const int64_t* __restrict__ cell_off, const CellGeom* __restrict__ geom,
                                                            Coefficient kc, double* kn )
{
   const int      z = blockIdx.x, c = blockIdx.y;
   const CellGeom g = geom[c];
   for ( int y = threadIdx.x; y + z <= ns; y += blockDim.x )
      for ( int x = 0; x + y + z <= ns; ++x )
      {
         double X[3], F[3], DF[3][3];
         for ( int d = 0; d < 3; ++d )
            X[d] = g.P[0][d] + ( ( g.P[1][d] - g.P[0][d] ) * x + ( g.P[2][d] - g.P[0][d] ) * y + ( g.P[3][d] - g.P[0][d] ) * z ) / double( ns );
         if ( g.blend == 1 ) shell_map( g, X, F, DF );
         else
            for ( int d = 0; d < 3; ++d ) F[d] = X[d];
         kn[cell_off[c] + cidx( ns, x, y, z )] = coeff_eval( kc, F );
      }
}

static void upload_geometry( Operator* op )
{
   if ( op->d_geom ) return;
   TableArrays arrays;
   CellGeom*   d_geom = arrays.upload( op->geom.data(), op->geom.size(), "geometry" );
   arrays.keep();
   op->d_geom = d_geom;
}

void set_p2_nodal_coefficient( Context* ctx, Operator* op, int Ls, const double* src )
{
   Mesh*    m = op->mesh;
   P1Level& P = m->level( Ls );
   ensure_device( m, P );
   upload_geometry( op );
   ElemLevel& e = op->el[Ls];
   if ( !e.d_kn ) check_cuda( cudaMalloc( &e.d_kn, P.size * sizeof( double ) ), "cudaMalloc(nodal coefficient)" );
   check_cuda( cudaMemsetAsync( e.d_kn, 0, P.size * sizeof( double ), ctx->stream ), "cudaMemset(nodal coefficient)" );
   if ( src )
      check_cuda( cudaMemcpyAsync( e.d_kn, src, P.size * sizeof( double ), cudaMemcpyDeviceToDevice, ctx->stream ), "copy nodal coefficient" );
   else
   {
      const dim3 grid( P.n + 1, m->topo.nC );
      k_p2_nodal_coeff<<< grid, 128, 0, ctx->stream >>>( P.n, P.d_off + P.nB, op->d_geom, op->coeff, e.d_kn );
      ++ctx->launches;
      check_cuda( cudaGetLastError(), "nodal coefficient launch" );
   }
}

// coordinates of a macro-cell's points in storage order (shared by all cells of the level)
static void ensure_cell_points( ElemLevel& e, const P1Level& P )
{
   if ( e.d_pts ) return;
   std::vector< ushort4 > pts;
   pts.reserve( size_t( tet_size( P.n + 1 ) ) );
   for ( int z = 0; z <= P.n; ++z )
      for ( int y = 0; y + z <= P.n; ++y )
         for ( int x = 0; x + y + z <= P.n; ++x ) pts.push_back( make_ushort4( (unsigned short) x, (unsigned short) y, (unsigned short) z, 0 ) );
   TableArrays arrays;
   ushort4*    d_pts = arrays.upload( pts.data(), pts.size(), "cell points" );
   arrays.keep();
   e.d_pts = d_pts;
}

// out[i + (i / block) (stride - block)] = in[i], rounded: one entry after the other of a slab of macro-cells into
// the level's weights
__global__ void __launch_bounds__( 256 ) k_slab_weights( int64_t count, int64_t block, int64_t stride, const double* __restrict__ in,
                                                          float* __restrict__ out )
{
   const int64_t i = int64_t( blockIdx.x ) * 256 + threadIdx.x;
   if ( i < count ) out[i + i / block * ( stride - block )] = float( in[i] );
}

// FP64 weights that the FP32 ones of a level are rounded from, at a time: with all of them beside the FP32 ones
// (230 + 115 bytes per node) the set-up needed twice the memory of FP32 element matrices, and levels that had
// fitted did not
constexpr int64_t kSlabBytes = int64_t( 256 ) << 20;

// FP32 weights of a P2 level, macro-cells in slabs of kSlabBytes (one cell at least)
static void fill_low_weights( Context* ctx, Mesh* m, Operator* op, int L, const P2StoredView& v, int64_t count, float* out )
{
   const int64_t per   = count / v.nC;  // weights of a macro-cell
   const int     cells = int( std::max< int64_t >( 1, std::min< int64_t >( v.nC, kSlabBytes / ( 8 * per ) ) ) );
   TableArrays   arrays;
   double*       slab = arrays.get< double >( per * cells, "stencil slab" );
   for ( int c0 = 0; c0 < v.nC; c0 += cells )
   {
      P2StoredView w = v;
      w.nC           = std::min( cells, v.nC - c0 );
      for ( int s = 0; s < 16; ++s ) w.wbase[s] = v.wbase[s] / v.nC * w.nC;
      check_cuda( cudaMemsetAsync( slab, 0, per * w.nC * sizeof( double ), ctx->stream ), "cudaMemset" );
      run_passes< double, double, 2 >( ctx, m, op, L, nullptr, nullptr, slab, &w, per * w.nC, c0 );
      for ( int s = 0; s < 16; ++s )
      {
         const int64_t n = ( s < 15 ? w.wbase[s + 1] : per * w.nC ) - w.wbase[s], block = int64_t( w.nC ) * v.np[s];
         if ( n == 0 ) continue;
         k_slab_weights<<< unsigned( ( n + 255 ) / 256 ), 256, 0, ctx->stream >>>( n, block, int64_t( v.nC ) * v.np[s], slab + w.wbase[s],
                                                                                   out + v.wbase[s] + int64_t( c0 ) * v.np[s] );
         ++ctx->launches;
      }
   }
   check_cuda( cudaGetLastError(), "stencil slab launch" );
   check_cuda( cudaStreamSynchronize( ctx->stream ), "stencil slabs" );
}

template < typename T, typename A >
static void ensure_level_t( Context* ctx, Operator* op, int L, int dtype )
{
   Mesh*    m = op->mesh;
   P1Level& P = m->level( L );
   ensure_device( m, P );
   upload_geometry( op );
   ensure_rows( op, L );
   ElemLevel& e = op->el[L];
   A*         acc = acc_buffer< A >( op, L, P.size );
   if ( op->store_matrices && op->order == 1 )
   {
      // P1: the stored matrices are kept assembled, summed in double once and rounded for float
      ensure_var_tables();
      const int64_t cnt = int64_t( 8 ) * P.size;
      ensure_cell_points( e, P );
      if ( !e.d_S[0] )
      {
         TableArrays arrays;
         double*     S = arrays.get< double >( cnt, "assembled stencils" );
         check_cuda( cudaMemsetAsync( S, 0, cnt * sizeof( double ), ctx->stream ), "cudaMemset" );
         run_passes< double, double, 4 >( ctx, m, op, L, nullptr, nullptr, S );
         arrays.keep();
         e.d_S[0] = S;
      }
      if ( sizeof( A ) == 4 && !e.d_S[1] )
      {
         TableArrays arrays;
         float*      S = arrays.get< float >( cnt, "assembled stencils" );
         launch_convert( ctx, cnt, F32, S, F64, e.d_S[0] );
         arrays.keep();
         e.d_S[1] = S;
      }
   }
   else if ( op->store_matrices && !e.d_S[sizeof( A ) == 8 ? 0 : 1] )
   {
      // P2: likewise; float weights alone are rounded from slabs of sums in double
      if ( !e.p2s )
      {
         std::vector< ushort4 > pts;
         std::vector< int >     rank;
         TableArrays            arrays;
         auto                   v     = std::make_shared< P2StoredView >();
         const int64_t          count = build_p2_stored( *v, P.n, m->topo.nC, pts, rank );
         ushort4*               d_pts  = arrays.upload( pts.data(), pts.size(), "stencil nodes" );
         int*                   d_rank = arrays.upload( rank.data(), rank.size(), "stencil ranks" );
         arrays.keep();
         v->pts       = d_pts;
         v->rank      = d_rank;
         e.d_p2s_pts  = d_pts;
         e.d_p2s_rank = d_rank;
         e.p2s_count  = count;
         e.p2s        = v;
      }
      TableArrays arrays;
      if ( sizeof( A ) == 8 )
      {
         double* S = arrays.get< double >( e.p2s_count, "assembled stencils" );
         check_cuda( cudaMemsetAsync( S, 0, e.p2s_count * sizeof( double ), ctx->stream ), "cudaMemset" );
         run_passes< double, double, 2 >( ctx, m, op, L, nullptr, nullptr, S, e.p2s.get(), e.p2s_count );
         arrays.keep();
         e.d_S[0] = S;
      }
      else
      {
         float* S = arrays.get< float >( e.p2s_count, "assembled stencils" );
         if ( e.d_S[0] ) launch_convert( ctx, e.p2s_count, F32, S, F64, e.d_S[0] );
         else fill_low_weights( ctx, m, op, L, *e.p2s, e.p2s_count, S );
         arrays.keep();
         e.d_S[1] = S;
      }
   }
   if ( e.d_invd[dtype] ) return;
   TableArrays arrays;
   A*          invd = arrays.get< A >( P.size, "inverse diagonal" );
   check_cuda( cudaMemsetAsync( invd, 0, P.size * sizeof( A ), ctx->stream ), "cudaMemset" );
   // diagonal: sum of element-matrix diagonals, owners summing their cell copies
   run_passes< T, A, 1 >( ctx, m, op, L, nullptr, acc );
   const int nrows = int( P.rows.size() );
   if ( nrows > 0 )
   {
      dim3 grid( ( nrows + 7 ) / 8, m->topo.nC );
      k_cell_invert< A ><<< grid, 256, 0, ctx->stream >>>( P.n, nrows, P.d_rows, P.d_off + P.nB, acc, invd );
   }
   if ( !P.tasks.empty() )
      launch_bnd_acc< T, A, OP_APPLY >( ctx, ctx->stream, P, kAll, 0, acc_vecs< T, A >( acc, {} ), 1, nullptr, invd, A( 0 ), A( 0 ) );
   check_cuda( cudaGetLastError(), "diagonal launch" );
   arrays.keep();
   e.d_invd[dtype] = invd;
}

void ensure_elementwise_level( Context* ctx, Operator* op, int L, int dtype )
{
   if ( dtype == F64 ) ensure_level_t< double, double >( ctx, op, L, dtype );
   else if ( dtype == F32 ) ensure_level_t< float, float >( ctx, op, L, dtype );
   else ensure_level_t< __half, float >( ctx, op, L, dtype );
}

template < typename T, typename A, int OP >
static void run_var( Context* ctx, Mesh* m, Operator* op, int L, int dtype, const StencilArgs& a )
{
   P1Level& P = m->level( L );
   ElemLevel& e  = op->el[L];
   A*         acc = acc_buffer< A >( op, L, P.size );
   const A*   S   = assembled_stencils< A >( op, L );
   const A*   inv = reinterpret_cast< const A* >( e.d_invd[dtype] );
   if ( P.n <= 2 )
   {
      const LevelView   v   = make_view( m, L );
      const BndSegments seg = bnd_segments( v, a.flag, a.copy_unflagged );
      if ( seg.threads == 0 ) return;
      k_var_low< T, A, OP ><<< ( seg.threads + 255 ) / 256, 256, 0, ctx->stream >>>( v, seg, a.flag, a.copy_unflagged, S, P.size, inv,
                                                                                     (const T*) a.src, (const T*) a.v1, (T*) a.v2,
                                                                                     (T*) a.dst, A( a.a0 ), A( a.a1 ) );
      ++ctx->launches;
      check_cuda( cudaGetLastError(), "assembled stencil launch" );
      return;
   }
   const int  np = int( tet_size( P.n + 1 ) ), stride = ( np + 31 ) / 32 * 32, nC = m->topo.nC;
   k_var_sweep< T, A, OP ><<< unsigned( ( int64_t( nC ) * stride + 255 ) / 256 ), 256, 0, ctx->stream >>>(
       P.n, nC, np, stride, reinterpret_cast< const ushort4* >( e.d_pts ), P.d_off + P.nB, P.d_bc + P.nB, a.flag, S, P.size, inv, acc,
       (const T*) a.src, (const T*) a.v1, (T*) a.v2, (T*) a.dst, A( a.a0 ), A( a.a1 ) );
   ++ctx->launches;
   launch_bnd_acc< T, A, OP >( ctx, ctx->stream, P, a.flag, a.copy_unflagged, acc_vecs< T, A >( acc, a ), 1, inv, nullptr, A( a.a0 ), A( a.a1 ) );
   check_cuda( cudaGetLastError(), "assembled stencil launch" );
}

// P2 level 0 with stored matrices, up to three components in one launch
template < typename T, typename A, int OP >
static void run_stored_low( Context* ctx, Mesh* m, Operator* op, int L, const A* S, const A* inv, const AccVecs< T, A >& vec, int ncomp,
                            const StencilArgs& a )
{
   const LevelView   v   = make_view( m, L );
   const BndSegments seg = bnd_segments( v, a.flag, a.copy_unflagged );
   if ( seg.threads == 0 ) return;
   k_p2_stored_low< T, A, OP ><<< dim3( ( seg.threads + 255 ) / 256, ncomp ), 256, 0, ctx->stream >>>(
       v, seg, *op->el[L].p2s, a.flag, a.copy_unflagged, S, inv, vec, A( a.a0 ), A( a.a1 ) );
   ++ctx->launches;
   check_cuda( cudaGetLastError(), "stored P2 launch" );
}

template < typename T, typename A, int OP >
static void run_elem( Context* ctx, Mesh* m, Operator* op, int L, int dtype, const StencilArgs& a )
{
   if ( op->order == 1 && assembled_stencils< A >( op, L ) ) return run_var< T, A, OP >( ctx, m, op, L, dtype, a );
   P1Level& P   = m->level( L );
   A*       acc = acc_buffer< A >( op, L, P.size );
   const A* inv = reinterpret_cast< const A* >( op->el[L].d_invd[dtype] );
   if ( const A* S = assembled_stencils< A >( op, L ) )
   {
      if ( P.n == 2 ) return run_stored_low< T, A, OP >( ctx, m, op, L, S, inv, acc_vecs< T, A >( acc, a ), 1, a );
      launch_p2_stored_sweep( ctx, P, dtype, *op->el[L].p2s, S, inv, acc, &a, 1 );
      launch_bnd_acc< T, A, OP >( ctx, ctx->stream, P, a.flag, a.copy_unflagged, acc_vecs< T, A >( acc, a ), 1, inv, nullptr, A( a.a0 ),
                                  A( a.a1 ) );
      check_cuda( cudaGetLastError(), "stored P2 combine launch" );
      return;
   }
   run_passes< T, A, 0 >( ctx, m, op, L, (const T*) a.src, acc );
   {
      struct Join
      {
         Context* c;
         ~Join()
         {
            cudaEventRecord( c->ev_join, c->aux );
            cudaStreamWaitEvent( c->stream, c->ev_join, 0 );
         }
      };
      check_cuda( cudaEventRecord( ctx->ev_fork, ctx->stream ), "fork" );
      check_cuda( cudaStreamWaitEvent( ctx->aux, ctx->ev_fork, 0 ), "fork" );
      Join j{ ctx };
      launch_cell_acc< T, A, OP >( ctx, m, P, a.flag, acc_vecs< T, A >( acc, a ), 1, inv, A( a.a0 ), A( a.a1 ) );
      launch_bnd_acc< T, A, OP >( ctx, ctx->aux, P, a.flag, a.copy_unflagged, acc_vecs< T, A >( acc, a ), 1, inv, nullptr, A( a.a0 ),
                                  A( a.a1 ) );
   }
   check_cuda( cudaGetLastError(), "elementwise combine launch" );
}

template < typename T, typename A >
static void dispatch_elem( Context* ctx, Mesh* m, Operator* op, int L, int dtype, const StencilArgs& a )
{
   switch ( a.op )
   {
   case OP_APPLY: run_elem< T, A, OP_APPLY >( ctx, m, op, L, dtype, a ); break;
   case OP_APPLY_ADD: run_elem< T, A, OP_APPLY_ADD >( ctx, m, op, L, dtype, a ); break;
   case OP_RESID: run_elem< T, A, OP_RESID >( ctx, m, op, L, dtype, a ); break;
   case OP_JAC: run_elem< T, A, OP_JAC >( ctx, m, op, L, dtype, a ); break;
   case OP_CHEB0: run_elem< T, A, OP_CHEB0 >( ctx, m, op, L, dtype, a ); break;
   case OP_CHEBI: run_elem< T, A, OP_CHEBI >( ctx, m, op, L, dtype, a ); break;
   case OP_CHEBL: run_elem< T, A, OP_CHEBL >( ctx, m, op, L, dtype, a ); break;
   case OP_DINV_APPLY: run_elem< T, A, OP_DINV_APPLY >( ctx, m, op, L, dtype, a ); break;
   default: throw std::invalid_argument( "unknown operation" );
   }
}

// owner/copy combine of the accumulation arrays of ncomp components (cell-array slots) with the epilogue
// of OP: cell interiors on the main stream, face/edge/vertex owners (sum of their cell copies, written
// through) on the second stream
template < typename T, typename A, int OP >
static void combine_acc( Context* ctx, Mesh* m, int L, const AccVecs< T, A >& vec, int ncomp, uint32_t flag, const A* invd = nullptr, A a0 = A( 0 ) )
{
   P1Level& P = m->level( L );
   struct Join
   {
      Context* c;
      ~Join()
      {
         cudaEventRecord( c->ev_join, c->aux );
         cudaStreamWaitEvent( c->stream, c->ev_join, 0 );
      }
   };
   check_cuda( cudaEventRecord( ctx->ev_fork, ctx->stream ), "fork" );
   check_cuda( cudaStreamWaitEvent( ctx->aux, ctx->ev_fork, 0 ), "fork" );
   Join      j{ ctx };
   launch_cell_acc< T, A, OP >( ctx, m, P, flag, vec, ncomp, invd, a0, A( 0 ) );
   launch_bnd_acc< T, A, OP >( ctx, ctx->aux, P, flag, 0, vec, ncomp, invd, nullptr, a0, A( 0 ) );
   check_cuda( cudaGetLastError(), "combine launch" );
}

template < typename T, typename A >
static void run_stokes( Context* ctx, Operator* op, int Lp, int divt, const void* const* u, const void* p, void* const* dst_u, void* dst_p,
                        uint32_t flag, int add, const StokesUpdate* up )
{
   Mesh*      m  = op->mesh;
   const int  Ls = Lp + 1;
   P1Level&   PP = m->level( Lp );
   P1Level&   PU = m->level( Ls );
   ensure_device( m, PP );
   ensure_device( m, PU );
   ensure_p2_constants();
   ensure_stokes_constants();
   upload_geometry( op );
   ensure_rows( op, Ls );
   ElemLevel& e = op->el[Ls];
   if ( !e.d_sacc )
      check_cuda( cudaMalloc( &e.d_sacc, size_t( 3 * PU.size + PP.size ) * sizeof( double ) ), "cudaMalloc(Stokes scratch)" );
   A* acc_u = reinterpret_cast< A* >( e.d_sacc );
   A* acc_p = acc_u + 3 * PU.size;
   if ( divt ) check_cuda( cudaMemsetAsync( acc_u, 0, size_t( 3 * PU.size ) * sizeof( A ), ctx->stream ), "cudaMemset" );
   else check_cuda( cudaMemsetAsync( acc_p, 0, size_t( PP.size ) * sizeof( A ), ctx->stream ), "cudaMemset" );
   const int nC = m->topo.nC;
   CoupledArgs< T, A > v{};
   for ( int k = 0; k < 3; ++k )
   {
      v.u[k]   = u ? (const T*) u[k] : nullptr;
      v.acc[k] = divt ? acc_u + k * PU.size : nullptr;
   }
   v.p = (const T*) p;
   if ( !divt ) v.acc[0] = acc_p;
   for ( int pc = 0; pc < 8; ++pc )
   {
      const int na = e.aoff[pc + 1] - e.aoff[pc];
      if ( na <= 0 ) continue;
      const unsigned blocks = unsigned( ( int64_t( na ) * nC + 31 ) / 32 );
      if ( divt )
         k_coupled_pass< T, A, CPL_DIVT ><<< blocks, kCoupledThreads, 0, ctx->stream >>>( 1 << Lp, nC, na, e.d_anch + e.aoff[pc], PP.d_off + PP.nB,
                                                                                         PU.d_off + PU.nB, op->d_geom, op->coeff, v, PP.size,
                                                                                         PU.size, ctx->d_error );
      else
         k_coupled_pass< T, A, CPL_DIV ><<< blocks, kCoupledThreads, 0, ctx->stream >>>( 1 << Lp, nC, na, e.d_anch + e.aoff[pc], PP.d_off + PP.nB,
                                                                                        PU.d_off + PU.nB, op->d_geom, op->coeff, v, PP.size,
                                                                                        PU.size, ctx->d_error );
      ++ctx->launches;
   }
   check_cuda( cudaGetLastError(), "Stokes pass launch" );
   AccVecs< T, A > vec{};
   if ( divt )
   {
      for ( int k = 0; k < 3; ++k )
      {
         vec.acc[k] = acc_u + k * PU.size;
         vec.dst[k] = (T*) dst_u[k];
         vec.v1[k]  = up ? (const T*) up->b[k] : nullptr;
      }
      if ( up ) combine_acc< T, A, OP_RESID >( ctx, m, Ls, vec, 3, flag );
      else if ( add ) combine_acc< T, A, OP_APPLY_ADD >( ctx, m, Ls, vec, 3, flag );
      else combine_acc< T, A, OP_APPLY >( ctx, m, Ls, vec, 3, flag );
      return;
   }
   vec.acc[0] = acc_p;
   vec.dst[0] = (T*) dst_p;
   if ( up )
   {
      if constexpr ( std::is_same< T, A >::value )
      {
         vec.src[0] = vec.dst[0];
         vec.v1[0]  = (const T*) up->b[0];
         combine_acc< T, A, OP_JAC >( ctx, m, Lp, vec, 1, flag, (const A*) up->sinv, A( up->omega ) );
      }
      else
         throw std::invalid_argument( "the fused pressure update needs FP64 or FP32 storage" );
   }
   else if ( add ) combine_acc< T, A, OP_APPLY_ADD >( ctx, m, Lp, vec, 1, flag );
   else combine_acc< T, A, OP_APPLY >( ctx, m, Lp, vec, 1, flag );
}

void launch_stokes_div( Context* ctx, Operator* op, int Lp, int dtype, int divt, const void* const* u, const void* p, void* const* dst_u,
                        void* dst_p, uint32_t flag, int add, const StokesUpdate* up )
{
   if ( dtype == F64 ) run_stokes< double, double >( ctx, op, Lp, divt, u, p, dst_u, dst_p, flag, add, up );
   else if ( dtype == F32 ) run_stokes< float, float >( ctx, op, Lp, divt, u, p, dst_u, dst_p, flag, add, up );
   else run_stokes< __half, float >( ctx, op, Lp, divt, u, p, dst_u, dst_p, flag, add, up );
}

// ---------------------------------------------------------------------------------------------
// Full viscous velocity block (P2ElementwiseBlendingFullViscousOperator.hpp:34-68): block (i, j) is
// the form p2_full_stokesvar_{i}_{j}_blending_q3, int 2 mu eps(u) : eps(v) - (2/3) mu div u div v
// with mu evaluated at the blended point, Yu's 5-point degree-3 rule.  Applied matrix-free per
// micro-cell: at each point the velocity gradient g (g_ik = d u_i / d x_k) of the ten local nodes
// gives the stress s = w mu |det| (g + g^T - (2/3) tr(g) I), and node a of component i receives
// grad phi_a . s_i; gradients and pairings go through the four vertices as in k_p2_apply_pass, the
// node sums meet in shared memory (k_coupled_pass).  The diagonal pass sums w mu |det| (|grad phi_a|^2 + (1/3) (d_i phi_a)^2).  Same
// parity passes as the coupling blocks (anchors of one class share no P2 node).
// ---------------------------------------------------------------------------------------------
__constant__ double c_yu5_rgrad[5][10][3];

static void ensure_visc_constants()
{
   static PerDeviceOnce once;
   once.run( [] {
      const double lg[4][3] = { { -1, -1, -1 }, { 1, 0, 0 }, { 0, 1, 0 }, { 0, 0, 1 } };
      const int    ed[6][2] = { { 2, 3 }, { 1, 3 }, { 1, 2 }, { 0, 3 }, { 0, 2 }, { 0, 1 } };
      const double pts[5][3] = { { 0.25, 0.25, 0.25 },
                                 { 1.0 / 6.0, 1.0 / 6.0, 1.0 / 6.0 },
                                 { 0.5, 1.0 / 6.0, 1.0 / 6.0 },
                                 { 1.0 / 6.0, 0.5, 1.0 / 6.0 },
                                 { 1.0 / 6.0, 1.0 / 6.0, 0.5 } };
      double g[5][10][3];
      for ( int q = 0; q < 5; ++q )
      {
         const double lam[4] = { 1.0 - pts[q][0] - pts[q][1] - pts[q][2], pts[q][0], pts[q][1], pts[q][2] };
         for ( int i = 0; i < 4; ++i )
            for ( int d = 0; d < 3; ++d ) g[q][i][d] = ( 4.0 * lam[i] - 1.0 ) * lg[i][d];
         for ( int e = 0; e < 6; ++e )
            for ( int d = 0; d < 3; ++d )
               g[q][4 + e][d] = 4.0 * ( lam[ed[e][0]] * lg[ed[e][1]][d] + lam[ed[e][1]] * lg[ed[e][0]][d] );
      }
      check_cuda( cudaMemcpyToSymbol( c_yu5_rgrad, g, sizeof( g ) ), "viscous block constants" );
   } );
}

// diagonal of the full viscous block, one parity pass
template < typename A >
__global__ void __launch_bounds__( 128 ) k_visc_diagonal( int ne, int nanch, const int* __restrict__ anch, const int64_t* __restrict__ off_u,
                                                       const CellGeom* __restrict__ geom, Coefficient kc, A* acc0, A* acc1, A* acc2,
                                                       int64_t size_u, int* err )
{
   const int t = blockIdx.x * blockDim.x + threadIdx.x;
   const int c = blockIdx.y;
   if ( t >= nanch ) return;
   const int      a  = anch[t];
   const int      x = a & 1023, y = ( a >> 10 ) & 1023, z = a >> 20, ns = 2 * ne;
   const CellGeom&      g     = geom[c];
   const int64_t  bu = off_u[c];
   for ( int ty = 0; ty < 6; ++ty )
   {
      if ( x + y + z > ne - 1 - c_mc_shift[ty] ) continue;
      int V[4][3];
      for ( int m = 0; m < 4; ++m )
         for ( int d = 0; d < 3; ++d ) V[m][d] = ( d == 0 ? x : d == 1 ? y : z ) + c_mc_off[ty][m][d];
      int64_t iu[10];
      for ( int m = 0; m < 4; ++m ) iu[m] = bu + cidx( ns, 2 * V[m][0], 2 * V[m][1], 2 * V[m][2] );
      for ( int e = 0; e < 6; ++e )
      {
         const int ea = c_p2_edge[e][0], eb = c_p2_edge[e][1];
         iu[4 + e]    = bu + cidx( ns, V[ea][0] + V[eb][0], V[ea][1] + V[eb][1], V[ea][2] + V[eb][2] );
      }
      {
         bool bad = false;
         for ( int m = 0; m < 10; ++m ) bad |= iu[m] < 0 || iu[m] >= size_u;
         if ( bad )
         {
            atomicExch( err, 2 );
            continue;
         }
      }
      MicroCell< A > mc;
      micro_cell( g, ne, ty, x, y, z, mc );
      {
         A yl[3][10];
         for ( int k = 0; k < 3; ++k )
            for ( int j = 0; j < 10; ++j ) yl[k][j] = A( 0 );
         for ( int q = 0; q < 5; ++q )
         {
            A Mi[3][3], adet, Fq[3];
            mapped_point( g, mc.X0, mc.J, c_yu5_pts[q], Mi, adet, Fq );
            const A s = A( c_yu5_w[q] ) * coeff_eval( kc, Fq ) * adet;
            for ( int b = 0; b < 10; ++b )
            {
               A G[3];
               for ( int k = 0; k < 3; ++k )
                  G[k] = A( c_yu5_rgrad[q][b][0] ) * Mi[0][k] + A( c_yu5_rgrad[q][b][1] ) * Mi[1][k] + A( c_yu5_rgrad[q][b][2] ) * Mi[2][k];
               const A gg = G[0] * G[0] + G[1] * G[1] + G[2] * G[2];
               for ( int i = 0; i < 3; ++i ) yl[i][b] += s * ( gg + A( 1.0 / 3.0 ) * G[i] * G[i] );
            }
         }
         for ( int j = 0; j < 10; ++j )
         {
            acc0[iu[j]] += yl[0][j];
            acc1[iu[j]] += yl[1][j];
            acc2[iu[j]] += yl[2][j];
         }
      }
   }
}

template < typename T, typename A >
static void run_visc( Context* ctx, Operator* op, int Lp, int mode, const void* const* u, void* const* dst, uint32_t flag, int add )
{
   Mesh*     m  = op->mesh;
   const int Ls = Lp + 1;
   P1Level&  PU = m->level( Ls );
   ensure_device( m, PU );
   ensure_p2_constants();
   ensure_visc_constants();
   upload_geometry( op );
   ensure_rows( op, Ls );
   ElemLevel& e = op->el[Ls];
   if ( !e.d_sacc ) check_cuda( cudaMalloc( &e.d_sacc, size_t( 3 * PU.size ) * sizeof( double ) ), "cudaMalloc(viscous block scratch)" );
   A* acc = reinterpret_cast< A* >( e.d_sacc );
   check_cuda( cudaMemsetAsync( acc, 0, size_t( 3 * PU.size ) * sizeof( A ), ctx->stream ), "cudaMemset" );
   const int nC = m->topo.nC;
   CoupledArgs< T, A > v{};
   for ( int k = 0; k < 3; ++k )
   {
      v.u[k]   = u ? (const T*) u[k] : nullptr;
      v.acc[k] = acc + k * PU.size;
   }
   for ( int pc = 0; pc < 8; ++pc )
   {
      const int na = e.aoff[pc + 1] - e.aoff[pc];
      if ( na <= 0 ) continue;
      if ( mode == 0 )
         k_coupled_pass< T, A, CPL_VISCOUS ><<< unsigned( ( int64_t( na ) * nC + 31 ) / 32 ), kCoupledThreads, 0, ctx->stream >>>(
             1 << Lp, nC, na, e.d_anch + e.aoff[pc], nullptr, PU.d_off + PU.nB, op->d_geom, op->coeff, v, 0, PU.size, ctx->d_error );
      else
      {
         const int bs = pass_block( na, 128 );
         dim3      grid( ( na + bs - 1 ) / bs, nC );
         k_visc_diagonal< A ><<< grid, bs, 0, ctx->stream >>>( 1 << Lp, na, e.d_anch + e.aoff[pc], PU.d_off + PU.nB, op->d_geom, op->coeff, acc,
                                                               acc + PU.size, acc + 2 * PU.size, PU.size, ctx->d_error );
      }
      ++ctx->launches;
   }
   check_cuda( cudaGetLastError(), "viscous block pass launch" );
   if ( mode == 0 )
   {
      AccVecs< T, A > vec{};
      for ( int k = 0; k < 3; ++k )
      {
         vec.acc[k] = acc + k * PU.size;
         vec.dst[k] = (T*) dst[k];
      }
      if ( add ) combine_acc< T, A, OP_APPLY_ADD >( ctx, m, Ls, vec, 3, flag );
      else combine_acc< T, A, OP_APPLY >( ctx, m, Ls, vec, 3, flag );
      return;
   }
   // diagonal: owners sum their copies, then 1/diag on every owned node (dst: three A arrays)
   const int nrows = int( PU.rows.size() );
   for ( int k = 0; k < 3; ++k )
   {
      A* invd = reinterpret_cast< A* >( dst[k] );
      check_cuda( cudaMemsetAsync( invd, 0, size_t( PU.size ) * sizeof( A ), ctx->stream ), "cudaMemset" );
      if ( nrows > 0 )
      {
         dim3 grid( ( nrows + 7 ) / 8, nC );
         k_cell_invert< A ><<< grid, 256, 0, ctx->stream >>>( PU.n, nrows, PU.d_rows, PU.d_off + PU.nB, acc + k * PU.size, invd );
      }
      if ( !PU.tasks.empty() )
         launch_bnd_acc< T, A, OP_APPLY >( ctx, ctx->stream, PU, kAll, 0, acc_vecs< T, A >( acc + k * PU.size, {} ), 1, nullptr, invd, A( 0 ),
                                           A( 0 ) );
   }
   check_cuda( cudaGetLastError(), "viscous block diagonal launch" );
}

void launch_full_viscous( Context* ctx, Operator* op, int Lp, int dtype, int mode, const void* const* u, void* const* dst, uint32_t flag,
                          int add )
{
   if ( dtype == F64 ) run_visc< double, double >( ctx, op, Lp, mode, u, dst, flag, add );
   else if ( dtype == F32 ) run_visc< float, float >( ctx, op, Lp, mode, u, dst, flag, add );
   else run_visc< __half, float >( ctx, op, Lp, mode, u, dst, flag, add );
}

template < typename T, typename A, int OP >
static void run_stored3( Context* ctx, Mesh* m, Operator* op, int L, int dtype, const StencilArgs* a )
{
   P1Level&   P = m->level( L );
   ElemLevel& e = op->el[L];
   const A*   S = assembled_stencils< A >( op, L );
   const A*   inv = reinterpret_cast< const A* >( e.d_invd[dtype] );
   if ( !e.d_sacc ) check_cuda( cudaMalloc( &e.d_sacc, size_t( 3 * P.size ) * sizeof( double ) ), "cudaMalloc(component scratch)" );
   A* acc = reinterpret_cast< A* >( e.d_sacc );
   AccVecs< T, A > vec{};
   for ( int k = 0; k < 3; ++k )
   {
      const AccVecs< T, A > v = acc_vecs< T, A >( acc + k * P.size, a[k] );
      vec.acc[k] = v.acc[0], vec.src[k] = v.src[0], vec.v1[k] = v.v1[0], vec.v2[k] = v.v2[0], vec.dst[k] = v.dst[0];
   }
   if ( P.n == 2 ) return run_stored_low< T, A, OP >( ctx, m, op, L, S, inv, vec, 3, a[0] );
   launch_p2_stored_sweep( ctx, P, dtype, *e.p2s, S, inv, acc, a, 3 );
   launch_bnd_acc< T, A, OP >( ctx, ctx->stream, P, a[0].flag, a[0].copy_unflagged, vec, 3, inv, nullptr, A( a[0].a0 ), A( a[0].a1 ) );
   check_cuda( cudaGetLastError(), "stored P2 combine launch" );
}

template < typename T, typename A >
static void dispatch_stored3( Context* ctx, Mesh* m, Operator* op, int L, int dtype, const StencilArgs* a )
{
   switch ( a[0].op )
   {
   case OP_CHEB0: run_stored3< T, A, OP_CHEB0 >( ctx, m, op, L, dtype, a ); break;
   case OP_CHEBI: run_stored3< T, A, OP_CHEBI >( ctx, m, op, L, dtype, a ); break;
   case OP_CHEBL: run_stored3< T, A, OP_CHEBL >( ctx, m, op, L, dtype, a ); break;
   default: throw std::invalid_argument( "operation not provided for three components" );
   }
}

bool launch_stored3( Context* ctx, Mesh* m, Operator* op, int L, int dtype, const StencilArgs* a )
{
   if ( !op->elementwise || op->order != 2 || !op->store_matrices ) return false;
   ensure_elementwise_level( ctx, op, L, dtype );
   if ( dtype == F64 ) dispatch_stored3< double, double >( ctx, m, op, L, dtype, a );
   else if ( dtype == F32 ) dispatch_stored3< float, float >( ctx, m, op, L, dtype, a );
   else dispatch_stored3< __half, float >( ctx, m, op, L, dtype, a );
   return true;
}

void launch_elementwise( Context* ctx, Mesh* m, Operator* op, int L, int dtype, const StencilArgs& a )
{
   ensure_elementwise_level( ctx, op, L, dtype );
   if ( dtype == F64 ) dispatch_elem< double, double >( ctx, m, op, L, dtype, a );
   else if ( dtype == F32 ) dispatch_elem< float, float >( ctx, m, op, L, dtype, a );
   else dispatch_elem< __half, float >( ctx, m, op, L, dtype, a );
}

}  // namespace hyb
