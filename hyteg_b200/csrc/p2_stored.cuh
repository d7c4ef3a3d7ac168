// P2 operators with stored matrices, kept assembled: layout of the stencils and their class tables.
//
// A P2 node of storage coordinates (x, y, z) couples with the nodes of the micro-cells around it; the set
// of offsets depends only on the parity of its coordinates (eight classes of 19 to 65 entries, 28.75 on
// average).  The weights of a level are grouped into sixteen segments, the eight classes of the nodes inside
// a macro-cell and the eight of the nodes on its boundary, and inside a segment entry by entry over all
// nodes of all macro-cells, so that consecutive threads read consecutive weights whatever the number of
// macro-cells or the length of their rows.  Boundary nodes hold the partial stencil of their macro-cell.
#pragma once

#include "hyb_device.cuh"

namespace hyb {

// vertices of the six micro-cell types (coordinate d of vertex i), and the P2 element's edges
__host__ __device__ constexpr int micro_vertex( int ty, int i, int d )
{
   constexpr int v[6][4][3] = {
       { { 0, 0, 0 }, { 1, 0, 0 }, { 0, 1, 0 }, { 0, 0, 1 } }, { { 1, 0, 0 }, { 1, 1, 0 }, { 0, 1, 0 }, { 1, 0, 1 } },
       { { 1, 0, 0 }, { 0, 1, 0 }, { 1, 0, 1 }, { 0, 0, 1 } }, { { 1, 1, 0 }, { 1, 1, 1 }, { 0, 1, 1 }, { 1, 0, 1 } },
       { { 1, 0, 1 }, { 0, 1, 1 }, { 0, 0, 1 }, { 0, 1, 0 } }, { { 0, 1, 0 }, { 1, 1, 0 }, { 1, 0, 1 }, { 0, 1, 1 } } };
   return v[ty][i][d];
}
__host__ __device__ constexpr int p2_edge_vertex( int e, int k )
{
   constexpr int v[6][2] = { { 2, 3 }, { 1, 3 }, { 1, 2 }, { 0, 3 }, { 0, 2 }, { 0, 1 } };
   return v[e][k];
}

// coordinate d of node i of micro-cell type ty in its anchor's 3x3x3 nodes
__host__ __device__ constexpr int p2_local( int ty, int i, int d )
{
   return i < 4 ? 2 * micro_vertex( ty, i, d ) : micro_vertex( ty, p2_edge_vertex( i - 4, 0 ), d ) + micro_vertex( ty, p2_edge_vertex( i - 4, 1 ), d );
}

struct P2Stencil {
   int n = 0;
   int off[65][3] = {};
};

// offsets of class p = (x & 1) | (y & 1) << 1 | (z & 1) << 2, sorted by (z, y, x): entries of one row of
// nodes are consecutive
__host__ __device__ constexpr P2Stencil p2_stencil( int p )
{
   P2Stencil s;
   for ( int dz = -2; dz <= 2; ++dz )
      for ( int dy = -2; dy <= 2; ++dy )
         for ( int dx = -2; dx <= 2; ++dx )
         {
            bool found = false;
            for ( int ty = 0; ty < 6 && !found; ++ty )
               for ( int i = 0; i < 10 && !found; ++i )
               {
                  const int a = p2_local( ty, i, 0 ), b = p2_local( ty, i, 1 ), c = p2_local( ty, i, 2 );
                  if ( ( ( a & 1 ) | ( b & 1 ) << 1 | ( c & 1 ) << 2 ) != p ) continue;
                  for ( int j = 0; j < 10 && !found; ++j )
                     found = p2_local( ty, j, 0 ) - a == dx && p2_local( ty, j, 1 ) - b == dy && p2_local( ty, j, 2 ) - c == dz;
               }
            if ( found )
            {
               s.off[s.n][0] = dx;
               s.off[s.n][1] = dy;
               s.off[s.n][2] = dz;
               ++s.n;
            }
         }
   return s;
}

template < int P >
struct P2Class {
   static constexpr P2Stencil S = p2_stencil( P );
};

// segment s = class + 8 (on the macro-cell's boundary): nodes per macro-cell, first entry of the node
// table, first weight; weight d of node k of macro-cell c is wbase[s] + (d nC + c) np[s] + k
struct P2StoredView {
   int            n, nC;
   int            np[16];
   int            pbase[16];
   int64_t        wbase[16];
   const ushort4* pts;   // coordinates of every segment's nodes
   const int*     rank;  // cell-array index of a node -> its number in its segment
};

// the weights' position of node (x, y, z) of macro-cell c, and the distance between its entries
__device__ __forceinline__ int64_t p2_weight_at( const P2StoredView& v, int c, int x, int y, int z, int64_t& step )
{
   const bool bnd = x == 0 || y == 0 || z == 0 || x + y + z == v.n;
   const int  s   = ( ( x & 1 ) | ( y & 1 ) << 1 | ( z & 1 ) << 2 ) + ( bnd ? 8 : 0 );
   step           = int64_t( v.nC ) * v.np[s];
   return v.wbase[s] + int64_t( c ) * v.np[s] + v.rank[cidx( v.n, x, y, z )];
}

// tables of a storage level with n nodes per macro-edge; returns the number of weights
int64_t build_p2_stored( P2StoredView& v, int n, int nC, std::vector< ushort4 >& pts, std::vector< int >& rank );
// entry of node j in node i's stencil, every micro-cell type: ent[(10 ty + i) 10 + j]
void p2_stored_entries( int8_t ent[600] );

}  // namespace hyb
