// Index arithmetic and tables that kernels use without checks of their own, run on the host over every point of
// small levels: node windows, row shifts, the positions of stored P2 weights, the micro-cells' stencil entries.
#include "hyb_internal.hpp"
#include "p2_stored.cuh"

#include <algorithm>
#include <cstdio>
#include <utility>

using namespace hyb;

static int failures = 0;
static void expect( bool ok, const char* what, int n, int x, int y, int z )
{
   if ( ok ) return;
   if ( ++failures < 20 ) std::printf( "%s: n %d point %d %d %d\n", what, n, x, y, z );
}

// the window of an anchor: its last index is the largest of all its nodes, and inside the cell array
static void windows( int n, int span )
{
   for ( int z = 0; z < n; z += span )
      for ( int y = 0; y + z < n; y += span )
         for ( int x = 0; x + y + z < n; x += span )
         {
            const int room = n - x - y - z;
            int64_t   last = 0;
            for ( int c = 0; c <= span; ++c )
               for ( int b = 0; b <= span; ++b )
                  for ( int a = 0; a <= span; ++a )
                     if ( a + b + c <= room ) last = std::max( last, cidx( n, x + a, y + b, z + c ) );
            expect( window_last( n, x, y, z, span, room ) == last && last < tet_size( n + 1 ), "window", n, x, y, z );
         }
}

// one class of the stored P2 stencils: every entry's neighbour by row_shift, its weight inside the array and its own
template < int P, int... D >
static void stored_class( const P2StoredView& v, int64_t count, std::vector< char >& taken, int c, int x, int y, int z, int seg, int k,
                          std::integer_sequence< int, D... > )
{
   auto entry = [&]( auto d ) {
      constexpr int e = decltype( d )::value, dx = P2Class< P >::S.off[e][0], dy = P2Class< P >::S.off[e][1], dz = P2Class< P >::S.off[e][2];
      const int64_t at = v.wbase[seg] + ( int64_t( e ) * v.nC + c ) * v.np[seg] + k;
      expect( at >= 0 && at < count && !taken[at], "stored weight", v.n, x, y, z );
      if ( at >= 0 && at < count ) taken[at] = 1;
      const bool inside = x + dx >= 0 && y + dy >= 0 && z + dz >= 0 && x + y + z + dx + dy + dz <= v.n;
      expect( seg >= 8 || inside, "interior neighbour", v.n, x, y, z );
      if ( inside )
         expect( cidx( v.n, x, y, z ) + row_shift< dy, dz >( v.n, y, z ) + dx == cidx( v.n, x + dx, y + dy, z + dz ), "row shift", v.n, x, y, z );
   };
   ( entry( std::integral_constant< int, D >{} ), ... );
}

static void stored( int n, int nC )
{
   P2StoredView           v;
   std::vector< ushort4 > pts;
   std::vector< int >     rank;
   const int64_t          count = build_p2_stored( v, n, nC, pts, rank );
   std::vector< char >    taken( count );
   int64_t                nodes = 0;
   for ( int seg = 0; seg < 16; ++seg )
      for ( int k = 0; k < v.np[seg]; ++k, ++nodes )
      {
         const ushort4 p = pts.at( v.pbase[seg] + k );
         const int     x = p.x, y = p.y, z = p.z;
         const bool    bnd = x == 0 || y == 0 || z == 0 || x + y + z == n;
         expect( seg == ( ( x & 1 ) | ( y & 1 ) << 1 | ( z & 1 ) << 2 ) + ( bnd ? 8 : 0 ), "segment", n, x, y, z );
         expect( rank.at( cidx( n, x, y, z ) ) == k, "rank", n, x, y, z );
         for ( int c = 0; c < nC; ++c )
         {
#define HYB_CLASS( P ) \
   if ( ( seg & 7 ) == P ) stored_class< P >( v, count, taken, c, x, y, z, seg, k, std::make_integer_sequence< int, P2Class< P >::S.n >() );
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
      }
   expect( nodes == tet_size( n + 1 ), "nodes of all segments", n, 0, 0, 0 );
   for ( char t : taken ) expect( t != 0, "weight of no node", n, 0, 0, 0 );
}

// every pair of a micro-cell's nodes has an entry of the first node's class that leads to the second
static void entries()
{
   int8_t ent[600];
   p2_stored_entries( ent );
   for ( int ty = 0; ty < 6; ++ty )
      for ( int i = 0; i < 10; ++i )
         for ( int j = 0; j < 10; ++j )
         {
            int l[3], m[3];
            for ( int d = 0; d < 3; ++d ) l[d] = p2_local( ty, i, d ), m[d] = p2_local( ty, j, d );
            const P2Stencil s = p2_stencil( ( l[0] & 1 ) | ( l[1] & 1 ) << 1 | ( l[2] & 1 ) << 2 );
            const int       e = ent[( 10 * ty + i ) * 10 + j];
            expect( e >= 0 && e < s.n && s.off[e][0] == m[0] - l[0] && s.off[e][1] == m[1] - l[1] && s.off[e][2] == m[2] - l[2], "entry", ty, i, j, 0 );
         }
}

// the 15 directions of the linear stencils from every point (k_var_sweep, k_flat_stencil)
template < int... D >
static void linear( int n, std::integer_sequence< int, D... > )
{
   for ( int z = 0; z <= n; ++z )
      for ( int y = 0; y + z <= n; ++y )
         for ( int x = 0; x + y + z <= n; ++x )
         {
            auto direction = [&]( auto d ) {
               constexpr int e = decltype( d )::value, dx = StencilDir< e >::x, dy = StencilDir< e >::y, dz = StencilDir< e >::z;
               if ( x + dx < 0 || y + dy < 0 || z + dz < 0 || x + y + z + dx + dy + dz > n ) return;
               expect( cidx( n, x, y, z ) + row_shift< dy, dz >( n, y, z ) + dx == cidx( n, x + dx, y + dy, z + dz ), "linear shift", n, x, y, z );
            };
            ( direction( std::integral_constant< int, D >{} ), ... );
         }
}

int main()
{
   for ( int n : { 1, 2, 4, 8, 16 } )
   {
      windows( n, 1 );
      if ( n > 1 ) windows( n, 2 );
      linear( n, std::make_integer_sequence< int, 15 >() );
      if ( n > 1 ) stored( n, n == 16 ? 1 : 3 );
   }
   entries();
   std::printf( failures ? "%d failures\n" : "index tables ok\n", failures );
   return failures != 0;
}
