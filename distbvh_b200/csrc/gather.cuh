// gather.cuh — the vertices of 32 elements from all over the vertex array into a warp's shared memory, by asynchronous
// copies in which neighbouring lanes copy neighbouring pieces of one element.
#pragma once

#include <cstdint>

#include "bulk_copy.cuh"

namespace bvhg {

// Shared-memory stride of one element's staged vertices, in doubles: elements of 4 and 8 vertices are padded by 16
// bytes, so that the 16-byte reads of 8 neighbouring threads fall into different banks (an odd stride of 9 doubles
// needs no padding).
template< int VT >
constexpr int kVertStride = VT == 0 ? 0 : ( VT % 2 == 0 ? VT * 3 + 2 : VT * 3 );

// LANES neighbouring lanes copy LANES neighbouring pieces (BYTES each, from piece FIRST on) of one of the 32 elements
// e (one per lane, the first `rows` of them): 32 / LANES elements per instruction, whose place needs no division.
template< int VT, int BYTES, int FIRST, int LANES >
__device__ __forceinline__ void gather_pieces(const double *__restrict__ verts, uint32_t e, int rows, double *s_v, int lane)
{
  constexpr int PER = 32 / LANES;
  const int w = ( FIRST + ( lane & ( LANES - 1 ) ) ) * ( BYTES / 8 ), q0 = lane / LANES;
#pragma unroll
  for ( int i = 0; i < LANES; ++i )
  {
    const int q = PER * i + q0;
    const uint32_t eq = __shfl_sync( 0xffffffffu, e, q );
    const double *src = verts + static_cast< size_t >( eq ) * ( VT * 3 ) + w;
    if ( q < rows )
    {
      if constexpr ( BYTES == 16 ) cp_async16( s_v + q * kVertStride< VT > + w, src );
      else cp_async_small< 8 >( s_v + q * kVertStride< VT > + w, src );
    }
  }
}

// The vertices of the 32 elements e into s_v by asynchronous copies.
template< int VT >
__device__ __forceinline__ void gather_vertices(const double *__restrict__ verts, uint32_t e, int rows, double *s_v, int lane)
{
  if constexpr ( VT % 2 == 0 )
  {
    // 6 or 12 pieces of 16 bytes
    if ( ( reinterpret_cast< uintptr_t >( verts ) & 15 ) == 0 )
    {
      if constexpr ( VT == 4 )
      {
        gather_pieces< VT, 16, 0, 4 >( verts, e, rows, s_v, lane );
        gather_pieces< VT, 16, 4, 2 >( verts, e, rows, s_v, lane );
      } else {
        gather_pieces< VT, 16, 0, 8 >( verts, e, rows, s_v, lane );
        gather_pieces< VT, 16, 8, 4 >( verts, e, rows, s_v, lane );
      }
      return;
    }
  }
  // 9, 12 or 24 pieces of 8 bytes
  gather_pieces< VT, 8, 0, 8 >( verts, e, rows, s_v, lane );
  if constexpr ( VT == 3 ) gather_pieces< VT, 8, 8, 1 >( verts, e, rows, s_v, lane );
  else if constexpr ( VT == 4 ) gather_pieces< VT, 8, 8, 4 >( verts, e, rows, s_v, lane );
  else
  {
    gather_pieces< VT, 8, 8, 8 >( verts, e, rows, s_v, lane );
    gather_pieces< VT, 8, 16, 8 >( verts, e, rows, s_v, lane );
  }
}

// This lane's staged vertices into registers.
template< int VT >
__device__ __forceinline__ void staged_vertices(const double *s_v, int q, double *v)
{
  const double *src = s_v + q * kVertStride< VT >;
  if constexpr ( VT % 2 == 0 )
  {
#pragma unroll
    for ( int k = 0; k < VT * 3; k += 2 )
    {
      const double2 t = *reinterpret_cast< const double2 * >( src + k );
      v[k] = t.x;
      v[k + 1] = t.y;
    }
  } else {
#pragma unroll
    for ( int k = 0; k < VT * 3; ++k ) v[k] = src[k];
  }
}

}  // namespace bvhg
