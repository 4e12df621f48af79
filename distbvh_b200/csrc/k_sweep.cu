// k_sweep.cu — sort-and-sweep candidate generation between two objects.
//
// Follows sort_and_sweep_local (src/bvh/narrowphase/kokkos.hpp:164-248) with the two objects as the two patches,
// and max_variant_axis (kokkos.hpp:125-160) for the sweep axis when the caller gives none:
// - the global range on the axis is the union of both objects' slab extents there (the K1 bounds of each object:
//   min of the cardinal slab minima, max of the maxima);
// - the reference scales B's slab minima on the axis to u32 keys, sorts them stably, and lets every element of A
//   sweep B in key order: it skips the B elements that end before its minimum, stops at the first that begins after
//   its maximum, and emits those that overlap it strictly on every slab. The emitted set is the exact pair set S(A, B)
//   for any axis.
// The emitted set is that of the strict all-slab overlap, so the order in which candidates are met is free. A one
// dimensional sweep of three dimensional elements meets thousands of them per element (two soups of 262,144 triangles:
// 4,000 B elements in every window). Here the sweep axis is cut into 256 strips and every strip is swept on a
// second axis (of the other two the one of larger extent), cut into 256 bins: B's key is (strip of its slab minimum,
// bin of its second slab minimum), 16 bits, two radix passes, and start[] holds the first sorted position of every
// (strip, bin) cell. An element of A then sweeps, in each strip of [its minimum - W, its maximum], the positions of
// the bins of [its second minimum - W2, its second maximum], where W and W2 are the largest widths of a B element on
// the two axes. Every overlapping B element lies there: b.min < a.max, and b.min >= b.max - W > a.min - W, with W
// rounded up, a.min - W rounded down and the strip a monotone function of the value. The candidates are tested on the
// third axis first, whose slabs lie contiguously in sorted order, then on the other slabs. The call on those two soups
// takes 0.40 ms instead of 4.46 ms.
// A degenerate axis (global_max == global_min) puts every element into strip or bin 0.
#include "bvhg_internal.cuh"
#include "kdop_math.cuh"

namespace bvhg {
int device_sm_count();
namespace {

constexpr int kSweepThreads = 256;
constexpr int kAxisBlocks = 512;  // partial sums of the axis choice (a fixed grid: a fixed summation order)

constexpr int kStrips = 256;  // strips of the sweep axis and bins of the second axis: one key byte each
constexpr int kCells = kStrips * kStrips;

struct sweep_params
{
  int axis;  // the sweep axis (read back by the host)
  int axis2, axis3;
  int pad;
  double gmin[2], fac[2];         // range minimum and scale factor of the sweep axis and the second axis
  unsigned long long wmax_enc[2]; // order-preserving encodings of W and W2
};

// Strip (or bin) of a value: monotone in v; NaN gives 0.
__device__ __forceinline__ uint32_t strip_of(double v, const sweep_params &p, int which)
{
  const double t = __dmul_rn( __dsub_rn( v, p.gmin[which] ), p.fac[which] );
  if ( !( t >= 0.0 ) ) return 0u;
  return t >= static_cast< double >( kStrips - 1 ) ? kStrips - 1 : static_cast< uint32_t >( t );
}

// The minimum and maximum of one coordinate over an element's vertices, with the inflation: the cardinal slab.
__device__ __forceinline__ void cardinal_slab(const double *__restrict__ src, int V, int axis, double eps, double &lo, double &hi)
{
  double mn = __ldg( src + axis ), mx = mn;
  for ( int v = 1; v < V; ++v )
  {
    const double t = __ldg( src + 3 * v + axis );
    mn = std_min( mn, t );
    mx = std_max( mx, t );
  }
  lo = __dsub_rn( mn, eps );
  hi = __dadd_rn( mx, eps );
}

// Partial sums of the centroids and their squares over A then B (block b: a grid-stride range), fixed order.
__global__ void __launch_bounds__( kSweepThreads ) k_axis_partial(const double *__restrict__ ax,
                                                                  const double *__restrict__ ay,
                                                                  const double *__restrict__ az, uint64_t na,
                                                                  const double *__restrict__ bx,
                                                                  const double *__restrict__ by,
                                                                  const double *__restrict__ bz, uint64_t nb,
                                                                  double *__restrict__ partial)
{
  __shared__ double s_red[6][kSweepThreads];
  double s[6] = { 0, 0, 0, 0, 0, 0 };
  const uint64_t n = na + nb;
  for ( uint64_t i = static_cast< uint64_t >( blockIdx.x ) * kSweepThreads + threadIdx.x; i < n;
        i += static_cast< uint64_t >( gridDim.x ) * kSweepThreads )
  {
    const double x = i < na ? ax[i] : bx[i - na];
    const double y = i < na ? ay[i] : by[i - na];
    const double z = i < na ? az[i] : bz[i - na];
    s[0] = __dadd_rn( s[0], x );
    s[1] = __dadd_rn( s[1], y );
    s[2] = __dadd_rn( s[2], z );
    s[3] = __dadd_rn( s[3], __dmul_rn( x, x ) );
    s[4] = __dadd_rn( s[4], __dmul_rn( y, y ) );
    s[5] = __dadd_rn( s[5], __dmul_rn( z, z ) );
  }
  for ( int k = 0; k < 6; ++k ) s_red[k][threadIdx.x] = s[k];
  __syncthreads();
  for ( int h = kSweepThreads / 2; h > 0; h >>= 1 )
  {
    if ( static_cast< int >( threadIdx.x ) < h )
      for ( int k = 0; k < 6; ++k ) s_red[k][threadIdx.x] = __dadd_rn( s_red[k][threadIdx.x], s_red[k][threadIdx.x + h] );
    __syncthreads();
  }
  if ( threadIdx.x < 6 ) partial[blockIdx.x * 6 + threadIdx.x] = s_red[threadIdx.x][0];
}

// The axis (given, or of largest centroid variance), the second axis, the global ranges on both and the scale
// factors. The partial sums are added in block order (one lane per sum, from shared memory: a single thread reading
// them from global memory took 135 us), so the axis does not depend on the run.
__global__ void __launch_bounds__( 256 ) k_sweep_setup(const double *__restrict__ partial, int nblocks, uint64_t n,
                                                       int axis_in, const obj_scalars *__restrict__ sa,
                                                       const obj_scalars *__restrict__ sb, sweep_params *__restrict__ p)
{
  __shared__ double s_part[kAxisBlocks * 6];
  __shared__ double s_sum[6];
  int axis = axis_in;
  if ( axis < 0 )
  {
    for ( int k = threadIdx.x; k < nblocks * 6; k += 256 ) s_part[k] = partial[k];
    __syncthreads();
    if ( threadIdx.x < 6 )
    {
      double s = 0;
      for ( int b = 0; b < nblocks; ++b ) s = __dadd_rn( s, s_part[b * 6 + threadIdx.x] );
      s_sum[threadIdx.x] = s;
    }
    __syncthreads();
  }
  if ( threadIdx.x != 0 ) return;
  if ( axis < 0 )
  {
    double var[3];
    for ( int k = 0; k < 3; ++k )
      var[k] = __dsub_rn( s_sum[3 + k], __ddiv_rn( __dmul_rn( s_sum[k], s_sum[k] ), static_cast< double >( n ) ) );
    axis = 0;
    if ( var[1] > var[0] ) axis = 1;
    if ( var[2] > var[axis] ) axis = 2;
  }
  double gmin[3], ext[3];
  for ( int k = 0; k < 3; ++k )
  {
    const double amin = ord_decode( sa->bounds_enc[k] ), amax = ord_decode( sa->bounds_enc[3 + k] );
    const double bmin = ord_decode( sb->bounds_enc[k] ), bmax = ord_decode( sb->bounds_enc[3 + k] );
    gmin[k] = bmin < amin ? bmin : amin;
    ext[k] = __dsub_rn( amax < bmax ? bmax : amax, gmin[k] );
  }
  const int u = axis == 0 ? 1 : 0, v = axis == 2 ? 1 : 2;  // the other two axes
  const int axis2 = ext[v] > ext[u] ? v : u;
  p->axis = axis;
  p->axis2 = axis2;
  p->axis3 = 3 - axis - axis2;
  p->gmin[0] = gmin[axis];
  p->gmin[1] = gmin[axis2];
  p->fac[0] = ext[axis] > 0.0 ? __ddiv_rn( static_cast< double >( kStrips ), ext[axis] ) : 0.0;
  p->fac[1] = ext[axis2] > 0.0 ? __ddiv_rn( static_cast< double >( kStrips ), ext[axis2] ) : 0.0;
  p->wmax_enc[0] = p->wmax_enc[1] = ord_encode( 0.0 );
}

// B's keys, the histograms of their two bytes, and the largest widths on the two axes.
__global__ void __launch_bounds__( kSweepThreads ) k_sweep_keys(const double *__restrict__ verts, int V, uint64_t n,
                                                                double eps, const sweep_params *pp,
                                                                uint64_t *__restrict__ keys, uint32_t *__restrict__ hist,
                                                                sweep_params *pw)  // pp and pw: the same struct
{
  __shared__ uint32_t s_hist[2 * 256];
  __shared__ double s_w[2][kSweepThreads / 32];
  for ( int k = threadIdx.x; k < 2 * 256; k += kSweepThreads ) s_hist[k] = 0;
  const sweep_params p = *pp;
  __syncthreads();
  const uint64_t i = static_cast< uint64_t >( blockIdx.x ) * kSweepThreads + threadIdx.x;
  double w[2] = { 0.0, 0.0 };
  if ( i < n )
  {
    const double *src = verts + i * V * 3;
    uint32_t key = 0;
#pragma unroll
    for ( int c = 0; c < 2; ++c )
    {
      double lo, hi;
      cardinal_slab( src, V, c ? p.axis2 : p.axis, eps, lo, hi );
      key = ( key << 8 ) | strip_of( lo, p, c );
      w[c] = __dsub_ru( hi, lo );
    }
    keys[i] = key;
    atomicAdd( &s_hist[key & 255u], 1u );
    atomicAdd( &s_hist[256 + ( key >> 8 )], 1u );
  }
#pragma unroll
  for ( int c = 0; c < 2; ++c )
  {
    for ( int o = 16; o > 0; o >>= 1 )
    {
      const double x = __shfl_xor_sync( 0xffffffffu, w[c], o );
      w[c] = w[c] > x ? w[c] : ( x > w[c] ? x : ( w[c] == w[c] ? w[c] : x ) );
    }
    if ( ( threadIdx.x & 31 ) == 0 ) s_w[c][threadIdx.x >> 5] = w[c];
  }
  __syncthreads();
  for ( int k = threadIdx.x; k < 2 * 256; k += kSweepThreads )
    if ( s_hist[k] ) atomicAdd( &hist[k], s_hist[k] );
  if ( threadIdx.x < 2 )
  {
    double m = 0.0;
    for ( int k = 0; k < kSweepThreads / 32; ++k ) m = s_w[threadIdx.x][k] > m ? s_w[threadIdx.x][k] : m;
    atomicMax( &pw->wmax_enc[threadIdx.x], ord_encode( m ) );
  }
}

// First index in [0, n) whose key is >= v.
__device__ __forceinline__ uint32_t key_bound(const uint64_t *__restrict__ keys, uint32_t n, uint32_t v)
{
  uint32_t lo = 0, hi = n;
  while ( lo < hi )
  {
    const uint32_t mid = ( lo + hi ) >> 1;
    if ( static_cast< uint32_t >( __ldg( keys + mid ) ) < v ) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

constexpr unsigned kStartBlocks = ( kCells + 1 + kSweepThreads - 1 ) / kSweepThreads;

// Blocks [0, kStartBlocks): start[c], the first sorted position of cell c or a later one (start[kCells] = n). The
// others: B's slabs in sorted order, slab by slab (the pair of slab a and position j at srows[2 (a n + j)]), so that
// a warp reads one slab of 32 neighbouring positions as one contiguous piece.
template< int K, int VT >
__global__ void __launch_bounds__( kSweepThreads ) k_sweep_gather(const double *__restrict__ verts, uint32_t Vrt,
                                                                  double eps, const uint64_t *__restrict__ skeys,
                                                                  const uint32_t *__restrict__ svals, uint64_t n,
                                                                  const obj_scalars *__restrict__ ssc,
                                                                  uint32_t *__restrict__ start,
                                                                  double *__restrict__ srows)
{
  constexpr int D = K / 2;
  if ( *reinterpret_cast< const volatile int * >( &ssc->error ) == kErrTimeout ) return;  // keys not sorted
  if ( blockIdx.x < kStartBlocks )
  {
    const uint32_t c = blockIdx.x * kSweepThreads + threadIdx.x;
    if ( c <= kCells ) start[c] = c == kCells ? static_cast< uint32_t >( n ) : key_bound( skeys, static_cast< uint32_t >( n ), c );
    return;
  }
  const uint64_t j = static_cast< uint64_t >( blockIdx.x - kStartBlocks ) * kSweepThreads + threadIdx.x;
  if ( j >= n ) return;
  double lo[D], hi[D];
  leaf_slabs< K, double, VT >( verts, Vrt, __ldg( svals + j ), eps, 0.f, lo, hi );
#pragma unroll
  for ( int a = 0; a < D; ++a )
    reinterpret_cast< double2 * >( srows )[static_cast< uint64_t >( a ) * n + j] = make_double2( lo[a], hi[a] );
}

constexpr int kPairThreads = 128;

// A: a warp takes `per` (at most 32) consecutive elements of A in Morton order. Every lane forms the slabs and the
// strip and bin ranges of one of them; then the warp sweeps them one after the other, 32 positions of a strip at a
// time. All lanes forming the same element's slabs, one warp per element, cost as much as the sweep itself.
template< int K, int VT >
__global__ void __launch_bounds__( kPairThreads ) k_sweep(const double *__restrict__ verts, uint32_t Vrt, uint64_t na,
                                                          uint32_t per, double eps, const sweep_params *__restrict__ pp,
                                                          const uint32_t *__restrict__ aperm,
                                                          const uint32_t *__restrict__ start,
                                                          const uint32_t *__restrict__ svals,
                                                          const double *__restrict__ srows, uint64_t nb,
                                                          const obj_scalars *__restrict__ ssc, uint2 *__restrict__ pairs,
                                                          uint64_t cap, pair_scalars *__restrict__ ps)
{
  constexpr int D = K / 2;
  __shared__ alignas( 16 ) double s_rows[kPairThreads / 32][32][K];
  if ( *reinterpret_cast< const volatile int * >( &ssc->error ) == kErrTimeout ) return;  // keys not sorted
  const sweep_params p = *pp;
  const unsigned lane = threadIdx.x & 31u, lt = ( 1u << lane ) - 1u;
  double( *rows )[K] = s_rows[threadIdx.x >> 5];
  const double2 *z = reinterpret_cast< const double2 * >( srows ) + static_cast< uint64_t >( p.axis3 ) * nb;
  const uint64_t first = static_cast< uint64_t >( ( blockIdx.x * kPairThreads + threadIdx.x ) >> 5 ) * per;
  uint32_t i = 0, span = 0;  // span: first strip, last strip, first bin, last bin
  if ( lane < per && first + lane < na )
  {
    i = __ldg( aperm + first + lane );
    double lo[D], hi[D];
    leaf_slabs< K, double, VT >( verts, Vrt, i, eps, 0.f, lo, hi );
#pragma unroll
    for ( int a = 0; a < D; ++a )
    {
      rows[lane][2 * a] = lo[a];
      rows[lane][2 * a + 1] = hi[a];
    }
#pragma unroll
    for ( int c = 0; c < 2; ++c )
    {
      const int a = c ? p.axis2 : p.axis;
      const double mn = a == 0 ? lo[0] : ( a == 1 ? lo[1] : lo[2] ), mx = a == 0 ? hi[0] : ( a == 1 ? hi[1] : hi[2] );
      span |= ( strip_of( __dsub_rd( mn, ord_decode( p.wmax_enc[c] ) ), p, c ) | ( strip_of( mx, p, c ) << 8 ) ) << ( 16 * c );
    }
  }
  __syncwarp();
  const uint32_t count = first < na ? static_cast< uint32_t >( min( static_cast< uint64_t >( per ), na - first ) ) : 0u;
  for ( uint32_t u = 0; u < count; ++u )
  {
    const uint32_t ai = __shfl_sync( 0xffffffffu, i, u ), sp = __shfl_sync( 0xffffffffu, span, u );
    const uint32_t s0 = sp & 255u, s1 = ( sp >> 8 ) & 255u, y0 = ( sp >> 16 ) & 255u, y1 = sp >> 24;
    const double *row = rows[u];
    const double zlo = row[2 * p.axis3], zhi = row[2 * p.axis3 + 1];
    for ( uint32_t sb = s0; sb <= s1; sb += 32 )
    {
      uint32_t b = 0, e = 0;  // the positions of strip sb + lane
      if ( sb + lane <= s1 )
      {
        b = __ldg( start + ( sb + lane ) * kStrips + y0 );
        e = __ldg( start + ( sb + lane ) * kStrips + y1 + 1 );
      }
      for ( unsigned m = __ballot_sync( 0xffffffffu, b < e ); m; m &= m - 1 )
      {
        const int s = __ffs( m ) - 1;
        const uint32_t jb = __shfl_sync( 0xffffffffu, b, s ), je = __shfl_sync( 0xffffffffu, e, s );
        for ( uint32_t j0 = jb; j0 < je; j0 += 32 )
        {
          const uint32_t j = j0 + lane;
          bool o = false;
          if ( j < je )
          {
            const double2 t = __ldg( z + j );
            o = zlo < t.y && t.x < zhi;
          }
          if ( !__any_sync( 0xffffffffu, o ) ) continue;
#pragma unroll 1
          for ( int a = 0; a < D; ++a )
          {
            if ( !o ) break;
            const double2 t = __ldg( reinterpret_cast< const double2 * >( srows ) + static_cast< uint64_t >( a ) * nb + j );
            o = row[2 * a] < t.y && t.x < row[2 * a + 1];
          }
          const unsigned bal = __ballot_sync( 0xffffffffu, o );
          if ( !bal ) continue;
          unsigned long long at = 0;
          if ( lane == 0 ) at = atomicAdd( &ps->count, static_cast< unsigned long long >( __popc( bal ) ) );
          at = __shfl_sync( 0xffffffffu, at, 0 ) + __popc( bal & lt );
          if ( o && at < cap ) pairs[at] = make_uint2( ai, __ldg( svals + j ) );
        }
      }
    }
  }
}

// Elements of A per warp: 32 when that still gives every SM 32 warps, fewer for a small A.
uint32_t sweep_per_warp(uint64_t na)
{
  const uint64_t warps = static_cast< uint64_t >( device_sm_count() ) * 32;
  const uint64_t per = na / warps;
  return static_cast< uint32_t >( per < 1 ? 1 : ( per > 32 ? 32 : per ) );
}

template< int K, int VT >
cudaError_t sweep_gather_t(const sweep_launch &x)
{
  const unsigned grid = kStartBlocks + static_cast< unsigned >( ( x.nb + kSweepThreads - 1 ) / kSweepThreads );
  k_sweep_gather< K, VT ><<< grid, kSweepThreads, 0, x.s >>>( x.bverts, x.bV, x.eps, x.skeys, x.svals, x.nb, x.sc, x.start, x.srows );
  return cudaGetLastError();
}

template< int K, int VT >
cudaError_t sweep_pairs_t(const sweep_launch &x)
{
  const uint32_t per = sweep_per_warp( x.na );
  const uint64_t warps = ( x.na + per - 1 ) / per;
  const unsigned grid = static_cast< unsigned >( ( warps + kPairThreads / 32 - 1 ) / ( kPairThreads / 32 ) );
  k_sweep< K, VT ><<< grid, kPairThreads, 0, x.s >>>( x.averts, x.aV, x.na, per, x.eps,
                                                     static_cast< const sweep_params * >( x.params ), x.aperm, x.start,
                                                     x.svals, x.srows, x.nb, x.sc, x.pairs, x.cap, x.ps );
  return cudaGetLastError();
}

template< int K >
cudaError_t sweep_k(const sweep_launch &x)
{
  cudaError_t e = cudaErrorInvalidValue;
  switch ( x.bV )
  {
    case 3: e = sweep_gather_t< K, 3 >( x ); break;
    case 4: e = sweep_gather_t< K, 4 >( x ); break;
    case 8: e = sweep_gather_t< K, 8 >( x ); break;
    default: e = sweep_gather_t< K, 0 >( x ); break;
  }
  if ( e != cudaSuccess ) return e;
  switch ( x.aV )
  {
    case 3: return sweep_pairs_t< K, 3 >( x );
    case 4: return sweep_pairs_t< K, 4 >( x );
    case 8: return sweep_pairs_t< K, 8 >( x );
    default: return sweep_pairs_t< K, 0 >( x );
  }
}

}  // namespace

size_t sweep_start_bytes() { return ( kCells + 1 ) * sizeof( uint32_t ); }
size_t sweep_params_bytes() { return sizeof( sweep_params ); }
size_t sweep_partial_bytes() { return static_cast< size_t >( kAxisBlocks ) * 6 * sizeof( double ); }

int sweep_axis_read(const void *params_host_copy) { return static_cast< const sweep_params * >( params_host_copy )->axis; }

cudaError_t launch_sweep_setup(const sweep_launch &x, int axis)
{
  if ( axis < 0 )
  {
    k_axis_partial<<< kAxisBlocks, kSweepThreads, 0, x.s >>>( x.acx, x.acy, x.acz, x.na, x.bcx, x.bcy, x.bcz, x.nb,
                                                             x.partial );
    cudaError_t e = cudaGetLastError();
    if ( e != cudaSuccess ) return e;
  }
  k_sweep_setup<<< 1, 256, 0, x.s >>>( x.partial, kAxisBlocks, x.na + x.nb, axis, x.asc, x.bsc,
                                       static_cast< sweep_params * >( x.params ) );
  return cudaGetLastError();
}

cudaError_t launch_sweep_keys(const sweep_launch &x)
{
  const unsigned grid = static_cast< unsigned >( ( x.nb + kSweepThreads - 1 ) / kSweepThreads );
  k_sweep_keys<<< grid, kSweepThreads, 0, x.s >>>( x.bverts, static_cast< int >( x.bV ), x.nb, x.eps,
                                                   static_cast< const sweep_params * >( x.params ), x.keys, x.hist,
                                                   static_cast< sweep_params * >( x.params ) );
  return cudaGetLastError();
}

cudaError_t launch_sweep(const sweep_launch &x)
{
  switch ( x.K )
  {
    case 6: return sweep_k< 6 >( x );
    case 18: return sweep_k< 18 >( x );
    case 26: return sweep_k< 26 >( x );
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace bvhg
