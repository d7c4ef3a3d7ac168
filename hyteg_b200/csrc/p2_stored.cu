// P2 operators with stored matrices: one gather sweep over the assembled stencils (layout: p2_stored.cuh).
#include "../../include/hyteg_b200.h"
#include "p2_stored.cuh"

#include <cuda_fp16.h>

#include <utility>

namespace hyb {

int64_t build_p2_stored( P2StoredView& v, int n, int nC, std::vector< ushort4 >& pts, std::vector< int >& rank )
{
   v    = P2StoredView{};
   v.n  = n;
   v.nC = nC;
   pts.clear();
   rank.assign( size_t( tet_size( n + 1 ) ), 0 );
   std::vector< ushort4 > seg[16];
   for ( int z = 0; z <= n; ++z )
      for ( int y = 0; y + z <= n; ++y )
         for ( int x = 0; x + y + z <= n; ++x )
         {
            const bool bnd = x == 0 || y == 0 || z == 0 || x + y + z == n;
            const int  s   = ( ( x & 1 ) | ( y & 1 ) << 1 | ( z & 1 ) << 2 ) + ( bnd ? 8 : 0 );
            rank[size_t( cidx( n, x, y, z ) )] = int( seg[s].size() );
            seg[s].push_back( make_ushort4( (unsigned short) x, (unsigned short) y, (unsigned short) z, 0 ) );
         }
   constexpr int entries[8] = { P2Class< 0 >::S.n, P2Class< 1 >::S.n, P2Class< 2 >::S.n, P2Class< 3 >::S.n,
                                P2Class< 4 >::S.n, P2Class< 5 >::S.n, P2Class< 6 >::S.n, P2Class< 7 >::S.n };
   int64_t       at         = 0;
   for ( int s = 0; s < 16; ++s )
   {
      v.np[s]    = int( seg[s].size() );
      v.pbase[s] = int( pts.size() );
      v.wbase[s] = at;
      at += int64_t( entries[s & 7] ) * nC * v.np[s];
      pts.insert( pts.end(), seg[s].begin(), seg[s].end() );
   }
   return at;
}

void p2_stored_entries( int8_t ent[600] )
{
   P2Stencil st[8];
   for ( int p = 0; p < 8; ++p ) st[p] = p2_stencil( p );
   for ( int ty = 0; ty < 6; ++ty )
      for ( int i = 0; i < 10; ++i )
      {
         int l[3];
         for ( int d = 0; d < 3; ++d ) l[d] = p2_local( ty, i, d );
         const P2Stencil& s = st[( l[0] & 1 ) | ( l[1] & 1 ) << 1 | ( l[2] & 1 ) << 2];
         for ( int j = 0; j < 10; ++j )
         {
            int e = 0;
            while ( e < s.n && ( s.off[e][0] != p2_local( ty, j, 0 ) - l[0] || s.off[e][1] != p2_local( ty, j, 1 ) - l[1] ||
                                 s.off[e][2] != p2_local( ty, j, 2 ) - l[2] ) )
               ++e;
            if ( e == s.n ) throw std::runtime_error( "P2 stencil tables: node pair not in its class" );
            ent[( 10 * ty + i ) * 10 + j] = int8_t( e );
         }
      }
}

namespace {

__device__ __forceinline__ double ldn( const double* p ) { return __ldg( p ); }
__device__ __forceinline__ float  ldn( const float* p ) { return __ldg( p ); }
__device__ __forceinline__ float  ldn( const __half* p ) { return __half2float( __ldg( p ) ); }
__device__ __forceinline__ double ldp( const double* p ) { return *p; }
__device__ __forceinline__ float  ldp( const float* p ) { return *p; }
__device__ __forceinline__ float  ldp( const __half* p ) { return __half2float( *p ); }
__device__ __forceinline__ void   stp( double* p, double v ) { *p = v; }
__device__ __forceinline__ void   stp( float* p, float v ) { *p = v; }
__device__ __forceinline__ void   stp( __half* p, float v ) { *p = __float2half_rn( v ); }
// weights are read once per sweep: they pass by L1, which keeps the vector
__device__ __forceinline__ double ldw( const double* p )
{
   double v;
   asm( "ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"( v ) : "l"( p ) );
   return v;
}
__device__ __forceinline__ float ldw( const float* p )
{
   float v;
   asm( "ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"( v ) : "l"( p ) );
   return v;
}

template < typename T, int NV >
struct StoredVecs {
   const T* src[NV];
   const T* v1[NV];
   T*       v2[NV];
   T*       dst[NV];
};

template < int P, bool BND, int D, typename T, typename A, int NV >
__device__ __forceinline__ void stored_term( const T* const ( &at )[NV], const A* W, int64_t step, int n, int x, int y, int z, A ( &s )[2][NV] )
{
   constexpr int dx = P2Class< P >::S.off[D][0], dy = P2Class< P >::S.off[D][1], dz = P2Class< P >::S.off[D][2];
   if ( BND )
      if ( x + dx < 0 || y + dy < 0 || z + dz < 0 || x + y + z + ( dx + dy + dz ) > n ) return;
   const A   w = ldw( W + D * step );
   const int o = row_shift< dy, dz >( n, y, z ) + dx;
#pragma unroll
   for ( int k = 0; k < NV; ++k ) s[D & 1][k] += w * A( ldn( at[k] + o ) );
}

template < int P, bool BND, typename T, typename A, int NV, int... D >
__device__ __forceinline__ void stored_terms( const T* const ( &at )[NV], const A* W, int64_t step, int n, int x, int y, int z, A ( &s )[2][NV],
                                              std::integer_sequence< int, D... > )
{
   ( stored_term< P, BND, D, T, A, NV >( at, W, step, n, x, y, z, s ), ... );
}

// One thread per node and all entries of its class unrolled, so the loads of a node are independent of
// each other.  Bound by the weights (230 bytes per node in FP64, read once, coalesced) and by the vector's
// rows, which every class reads from L2 again: element matrices took 330 bytes and eight passes of
// read-modify-writes over the nodes, and one launch replaces ten.  Chebyshev(3) step on a shell of 240 cells,
// level 4, FP64: 898 -> 430 us.  (A block per cell with the vector in shared memory: 519 us.)  Nodes inside a
// macro-cell finish here; those on its boundary leave their partial sums in acc, which the owners then
// combine.  With three vectors (the velocity components) the weights are read once for all.
template < typename T, typename A, int NV >
__global__ void __launch_bounds__( 256 )
    k_p2_stored_sweep( P2StoredView v, int op, uint32_t flag, const uint8_t* __restrict__ cell_bc, const int64_t* __restrict__ cell_off,
                       const A* __restrict__ S, const A* __restrict__ invd, StoredVecs< T, NV > vec, A* __restrict__ acc, int64_t acc_step,
                       A a0, A a1 )
{
   int     seg = 0;
   int64_t g   = blockIdx.x;
   for ( ; seg < 15; ++seg )
   {
      const int64_t blocks = ( int64_t( v.nC ) * v.np[seg] + 255 ) / 256;
      if ( g < blocks ) break;
      g -= blocks;
   }
   const int np = v.np[seg];
   g            = g * 256 + threadIdx.x;
   if ( g >= int64_t( v.nC ) * np ) return;
   const int c = g < 0x7fffffff ? int( unsigned( g ) / unsigned( np ) ) : int( g / np );
   if ( seg < 8 && !( cell_bc[c] & flag ) ) return;
   const ushort4 pt = v.pts[v.pbase[seg] + int( g - int64_t( c ) * np )];
   const int     x = pt.x, y = pt.y, z = pt.z, n = v.n;
   const int64_t i    = cell_off[c] + cidx( n, x, y, z );
   const int64_t step = int64_t( v.nC ) * np;
   const A*      W    = S + v.wbase[seg] + g;
   const T*      at[NV];
   A             s[2][NV];
#pragma unroll
   for ( int k = 0; k < NV; ++k )
   {
      at[k]   = vec.src[k] + i;
      s[0][k] = s[1][k] = A( 0 );
   }
   switch ( seg )
   {
#define HYB_CLASS( P )                                                                                                            \
   case P: stored_terms< P, false, T, A, NV >( at, W, step, n, x, y, z, s, std::make_integer_sequence< int, P2Class< P >::S.n >() ); break; \
   case P + 8: stored_terms< P, true, T, A, NV >( at, W, step, n, x, y, z, s, std::make_integer_sequence< int, P2Class< P >::S.n >() ); break;
      HYB_CLASS( 0 )
      HYB_CLASS( 1 )
      HYB_CLASS( 2 )
      HYB_CLASS( 3 )
      HYB_CLASS( 4 )
      HYB_CLASS( 5 )
      HYB_CLASS( 6 )
      HYB_CLASS( 7 )
#undef HYB_CLASS
   }
   if ( seg >= 8 )
   {
#pragma unroll
      for ( int k = 0; k < NV; ++k ) acc[k * acc_step + i] = s[0][k] + s[1][k];
      return;
   }
   const A di = op == OP_APPLY || op == OP_APPLY_ADD || op == OP_RESID ? A( 1 ) : invd[i];
#pragma unroll
   for ( int k = 0; k < NV; ++k )
   {
      const A  r   = s[0][k] + s[1][k];
      const T* src = vec.src[k] + i;
      const T* v1  = vec.v1[k] + i;
      T*       v2  = vec.v2[k] + i;
      T*       dst = vec.dst[k] + i;
      switch ( op )
      {
      case OP_APPLY: stp( dst, r ); break;
      case OP_APPLY_ADD: stp( dst, A( ldp( dst ) ) + r ); break;
      case OP_RESID: stp( dst, A( ldp( v1 ) ) - r ); break;
      case OP_JAC: stp( dst, A( ldp( src ) ) + a0 * ( di * ( A( ldp( v1 ) ) - r ) ) ); break;
      case OP_CHEB0: stp( dst, di * ( A( ldp( v1 ) ) - r ) ); break;
      case OP_CHEBI:
      {
         const A u = A( ldp( v2 ) ) + a0 * A( ldp( src ) );
         stp( dst, di * r );
         stp( v2, u );
         break;
      }
      case OP_CHEBL: stp( v2, ( A( ldp( v2 ) ) + a0 * A( ldp( src ) ) ) + a1 * ( di * r ) ); break;
      case OP_DINV_APPLY: stp( dst, di * r ); break;
      }
   }
}

template < typename T, typename A, int NV >
void run_sweep( Context* ctx, P1Level& P, const P2StoredView& v, const void* S, const void* invd, void* acc, const StencilArgs* a )
{
   int64_t blocks = 0;
   for ( int s = 0; s < 16; ++s ) blocks += ( int64_t( v.nC ) * v.np[s] + 255 ) / 256;
   if ( blocks == 0 ) return;
   StoredVecs< T, NV > vec;
   for ( int k = 0; k < NV; ++k )
   {
      vec.src[k] = (const T*) a[k].src;
      vec.v1[k]  = (const T*) a[k].v1;
      vec.v2[k]  = (T*) a[k].v2;
      vec.dst[k] = (T*) a[k].dst;
   }
   k_p2_stored_sweep< T, A, NV ><<< unsigned( blocks ), 256, 0, ctx->stream >>>( v, a[0].op, a[0].flag, P.d_bc + P.nB, P.d_off + P.nB,
                                                                                (const A*) S, (const A*) invd, vec, (A*) acc, P.size,
                                                                                A( a[0].a0 ), A( a[0].a1 ) );
   ++ctx->launches;
   check_cuda( cudaGetLastError(), "stored P2 sweep launch" );
}

}  // namespace

void launch_p2_stored_sweep( Context* ctx, P1Level& P, int dtype, const P2StoredView& v, const void* S, const void* invd, void* acc,
                             const StencilArgs* a, int ncomp )
{
   auto run = [&]( auto nv ) {
      constexpr int NV = decltype( nv )::value;
      if ( dtype == F64 ) run_sweep< double, double, NV >( ctx, P, v, S, invd, acc, a );
      else if ( dtype == F32 ) run_sweep< float, float, NV >( ctx, P, v, S, invd, acc, a );
      else run_sweep< __half, float, NV >( ctx, P, v, S, invd, acc, a );
   };
   if ( ncomp == 1 ) run( std::integral_constant< int, 1 >{} );
   else if ( ncomp == 3 ) run( std::integral_constant< int, 3 >{} );
   else throw std::invalid_argument( "stored P2 sweep: one or three vectors" );
}

}  // namespace hyb
