// k_sweep.cu — sort-and-sweep candidate generation between two objects.
//
// Follows sort_and_sweep_local (src/bvh/narrowphase/kokkos.hpp:164-248) with the two objects as the two patches,
// and max_variant_axis (kokkos.hpp:125-160) for the sweep axis when the caller gives none:
// the reference scales B's slab minima on the axis to u32 keys over the union of both objects' extents, sorts them
// stably, and lets every element of A sweep B in key order: it skips the B elements that end before its minimum, stops
// at the first that begins after its maximum, and emits those that overlap it strictly on every slab. The emitted set is
// the exact pair set S(A, B) for any axis.
// The emitted set is that of the strict all-slab overlap, so the order in which candidates are met is free. A one
// dimensional sweep of three dimensional elements meets thousands of them per element (two soups of 262,144 triangles:
// 4,000 B elements in every window). Here the sweep axis is cut into 256 strips and every strip is swept on a
// second axis (of the other two the one on which B's minima spread further), cut into 256 bins: B's key is (strip of its
// slab minimum, bin of its second slab minimum), 16 bits, two radix passes, and start[] holds the first sorted position
// of every (strip, bin) cell. An element of A then sweeps, in each strip of [its minimum - W, its maximum], the
// positions of the bins of [its second minimum - W2, its second maximum], where W and W2 are the largest widths of a B
// element on the two axes. Every overlapping B element lies there: b.min < a.max, and b.min >= b.max - W > a.min - W,
// with W rounded up, a.min - W rounded down and the strip a monotone function of the value. The candidates are tested on
// the third axis first, whose slabs lie contiguously in sorted order, then on the other slabs.
// The borders of the strips (and bins) follow B's elements wherever they lie: 32 quantiles of B's slab minima, from a
// sample of 1,024, and 8 even steps to the next one. A strip holds about nb / 256 elements, and a sweep meets at most two
// partial strips beyond the elements that a one dimensional window holds. (Even steps over the objects' extents took the
// same time for a uniform soup, but with one element 1,000 extents away nearly all of B lay in one cell and every element
// of A met all of it.) Two soups of 262,144 triangles, us per call, with one dimensional windows of 32-bit keys, with even
// steps, and now:
//   uniform                                        3,850     300     300
//   one element of B (or of A) 1,000 extents away  3,960 152,000     300
//   two clusters 30 extents apart                  2,190   1,730     267
//   normal deviates cubed                         11,900  54,000  11,200 (its dense middle holds most of the pairs)
//   A 100 times as wide and as coarse              6,150   6,300   2,600
#include "bvhg_internal.cuh"
#include "kdop_math.cuh"

namespace bvhg {
int device_sm_count();
namespace {

constexpr int kSweepThreads = 256;
constexpr int kAxisBlocks = 512;  // partial sums of the axis choice (a fixed grid: a fixed summation order)

constexpr int kStrips = 256;  // strips of the sweep axis and bins of the second axis: one key byte each
constexpr int kCells = kStrips * kStrips;
constexpr int kKnots = 32;            // quantiles per axis
constexpr int kSteps = kStrips / kKnots;  // strips between two of them
constexpr int kSample = 1024;         // minima sampled per axis for them

struct sweep_params
{
  int axis;  // the sweep axis (read back by the host)
  int pad;
  unsigned long long wmax_enc[2];  // order-preserving encodings of W and W2
  double knot[3][kKnots + 1];      // per axis: quantiles of B's slab minima, ascending
  int axis2, axis3;
  double2 cut[2][kKnots];          // of the sweep axis and the second axis: (knot, strips per unit after it)
};

// The second axis: of the other two the one on which the middle three quarters of B's minima spread further.
__device__ __forceinline__ int second_axis(const sweep_params *p, int axis)
{
  const int u = axis == 0 ? 1 : 0, v = axis == 2 ? 1 : 2;
  constexpr int q0 = kKnots / 8, q1 = kKnots - q0;
  return p->knot[v][q1] - p->knot[v][q0] > p->knot[u][q1] - p->knot[u][q0] ? v : u;
}

// Strip (or bin) of a value: monotone in v (NaN gives 0). Between two knots the strips are even steps; equal knots, whose
// strips per unit are infinite, and knots further apart than a double tells still give a step in [0, kSteps).
__device__ __forceinline__ uint32_t strip_between(double v, uint32_t q, double knot, double per_unit)
{
  const double t = __dmul_rn( __dsub_rn( v, knot ), per_unit );
  return q * kSteps + ( t > 0.0 ? ( t < static_cast< double >( kSteps ) ? static_cast< uint32_t >( t ) : kSteps - 1u ) : 0u );
}
__device__ __forceinline__ uint32_t strip_of(double v, const double *knot, const double *per_unit)
{
  uint32_t q = 0;
#pragma unroll
  for ( uint32_t step = kKnots / 2; step > 0; step >>= 1 )
    if ( knot[q + step] <= v ) q += step;
  return strip_between( v, q, knot[q], per_unit[q] );
}
// The same by a whole warp whose lane q holds knot q and the strips per unit after it.
__device__ __forceinline__ uint32_t strip_of(double v, double knot, double per_unit)
{
  static_assert( kKnots == 32, "one knot per lane" );
  uint32_t q = 0;
#pragma unroll
  for ( uint32_t step = kKnots / 2; step > 0; step >>= 1 )
    if ( __shfl_sync( 0xffffffffu, knot, q + step ) <= v ) q += step;
  return strip_between( v, q, __shfl_sync( 0xffffffffu, knot, q ), __shfl_sync( 0xffffffffu, per_unit, q ) );
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

// Blocks [0, 3 per): the knots of the three axes, per blocks each. The sample takes one element of each of cnt equal
// ranges of B (step elements each), its place in the range from a hash (an even stride would meet the same row of a
// lattice again and again). The sample is not sorted: every block reads all of its axis and ranks 32 of its minima, 8
// lanes per minimum and an eighth of the sample each, and the minima whose ranks are the quantiles write themselves. (A
// bitonic network over 2,048 minima in one block per axis made a call 28 us longer.)
// The other blocks (none when the caller gives the axis): partial sums of the centroids and their squares over A then B,
// a grid-stride range each, fixed order, and the axis of largest centroid variance from them.
constexpr int kRankLanes = 8;

__device__ __forceinline__ void set_axis(sweep_params *p, int axis)
{
  p->axis = axis;
  p->wmax_enc[0] = p->wmax_enc[1] = ord_encode( 0.0 );
}

__global__ void __launch_bounds__( kSweepThreads ) k_sweep_sample(sweep_launch x, int axis_in, int per, int cnt, double step)
{
  __shared__ alignas( 16 ) double s_val[6 * kSweepThreads];
  static_assert( kSample <= 6 * kSweepThreads, "one array for both" );
  const int t = threadIdx.x;
  if ( static_cast< int >( blockIdx.x ) < 3 * per )
  {
    if ( axis_in >= 0 && blockIdx.x == 0 && t == 0 ) set_axis( static_cast< sweep_params * >( x.params ), axis_in );
    const int k = blockIdx.x / per;
    const int V = static_cast< int >( x.bV );
    // a thread's samples together: one trip to memory per vertex
    constexpr int PER = kSample / kSweepThreads;
    const double *src[PER];
    double mn[PER];
#pragma unroll
    for ( int q = 0; q < PER; ++q )
    {
      const int j = q * kSweepThreads + t;
      src[q] = x.bverts + k;
      if ( j < cnt )
      {
        uint32_t h = static_cast< uint32_t >( j ) + 1u;  // a 32-bit mixer of shifts and odd multipliers
        h = ( h ^ ( h >> 16 ) ) * 0x7feb352du;
        h = ( h ^ ( h >> 15 ) ) * 0x846ca68bu;
        h ^= h >> 16;
        const uint64_t e = static_cast< uint64_t >( __dmul_rn( j + h * 0x1p-32, step ) );
        src[q] += min( e, x.nb - 1 ) * V * 3;
      }
      mn[q] = __ldg( src[q] );
    }
    for ( int v = 1; v < V; ++v )
    {
#pragma unroll
      for ( int q = 0; q < PER; ++q ) mn[q] = std_min( mn[q], __ldg( src[q] + 3 * v ) );
    }
#pragma unroll
    for ( int q = 0; q < PER; ++q ) s_val[q * kSweepThreads + t] = __dsub_rn( mn[q], x.eps );
    __syncthreads();
    // rank: the minima below it, and the equal ones before it
    const int i = ( static_cast< int >( blockIdx.x ) % per ) * ( kSweepThreads / kRankLanes ) + t / kRankLanes;
    const double mine = i < cnt ? s_val[i] : 0.0;
    int rank = 0;
#pragma unroll 8
    for ( int j = t % kRankLanes; j < cnt; j += kRankLanes )
    {
      const double y = s_val[j];
      rank += ( y < mine ) | ( ( y == mine ) & ( j < i ) );
    }
#pragma unroll
    for ( int o = 1; o < kRankLanes; o <<= 1 ) rank += __shfl_xor_sync( 0xffffffffu, rank, o );
    if ( i >= cnt || t % kRankLanes ) return;
    // knot q is the minimum of rank q cnt / kKnots (q of one rank: consecutive, none or several), the last the largest
    double *knot = static_cast< sweep_params * >( x.params )->knot[k];
    for ( int q = ( rank * kKnots + cnt - 1 ) / cnt; q < kKnots && q * cnt / kKnots == rank; ++q ) knot[q] = mine;
    if ( rank == cnt - 1 ) knot[kKnots] = mine;
    return;
  }
  const uint64_t block = blockIdx.x - 3 * per, na = x.na, n = x.na + x.nb;
  double s[6] = { 0, 0, 0, 0, 0, 0 };
  for ( uint64_t i = block * kSweepThreads + t; i < n; i += static_cast< uint64_t >( kAxisBlocks ) * kSweepThreads )
  {
    const double c[3] = { __ldg( i < na ? x.acx + i : x.bcx + ( i - na ) ), __ldg( i < na ? x.acy + i : x.bcy + ( i - na ) ),
                          __ldg( i < na ? x.acz + i : x.bcz + ( i - na ) ) };
#pragma unroll
    for ( int k = 0; k < 3; ++k )
    {
      s[k] = __dadd_rn( s[k], c[k] );
      s[3 + k] = __dadd_rn( s[3 + k], __dmul_rn( c[k], c[k] ) );
    }
  }
  for ( int k = 0; k < 6; ++k ) s_val[k * kSweepThreads + t] = s[k];
  __syncthreads();
  for ( int h = kSweepThreads / 2; h > 0; h >>= 1 )
  {
    if ( t < h )
      for ( int k = 0; k < 6; ++k )
        s_val[k * kSweepThreads + t] = __dadd_rn( s_val[k * kSweepThreads + t], s_val[k * kSweepThreads + t + h] );
    __syncthreads();
  }
  if ( t < 6 )
  {
    x.partial[block * 6 + t] = s_val[t * kSweepThreads];
    __threadfence();
  }
  __syncthreads();
  // the last block to finish chooses the axis: the sums are added in block order (one lane per sum, from shared memory: a
  // single thread reading them from global memory took 135 us), so it does not depend on the run
  __shared__ bool s_last;
  if ( t == 0 ) s_last = atomicAdd( x.hist + 2 * 256, 1u ) == kAxisBlocks - 1;
  __syncthreads();
  if ( !s_last ) return;
  __threadfence();
  __shared__ double s_part[kAxisBlocks * 6];
  for ( int k = t; k < kAxisBlocks * 6; k += kSweepThreads ) s_part[k] = __ldcg( x.partial + k );
  __syncthreads();
  if ( t < 6 )
  {
    double sum = 0;
#pragma unroll 4
    for ( int b = 0; b < kAxisBlocks; ++b ) sum = __dadd_rn( sum, s_part[b * 6 + t] );
    s_val[t] = sum;
  }
  __syncthreads();
  if ( t != 0 ) return;
  double var[3];
  for ( int k = 0; k < 3; ++k )
    var[k] = __dsub_rn( s_val[3 + k], __ddiv_rn( __dmul_rn( s_val[k], s_val[k] ), static_cast< double >( n ) ) );
  int axis = 0;
  if ( var[1] > var[0] ) axis = 1;
  if ( var[2] > var[axis] ) axis = 2;
  set_axis( static_cast< sweep_params * >( x.params ), axis );
}

// B's keys, the histograms of their two bytes, and the largest widths on the two axes. A grid of at most two blocks per
// SM strides over the elements: every block adds up to 512 counts to the histograms, and those atomics were most of the
// kernel with one block per 256 elements (262,144 elements 18.6 -> 12.1 us).
__global__ void __launch_bounds__( kSweepThreads ) k_sweep_keys(const double *__restrict__ verts, int V, uint64_t n,
                                                                double eps, const sweep_params *pp,
                                                                uint64_t *__restrict__ keys, uint32_t *__restrict__ hist,
                                                                sweep_params *pw)  // pp and pw: the same struct
{
  __shared__ uint32_t s_hist[2 * 256];
  __shared__ double s_knot[2][kKnots], s_per[2][kKnots];
  __shared__ double s_w[2][kSweepThreads / 32];
  const int axis = pp->axis, axis2 = second_axis( pp, axis );
  for ( int k = threadIdx.x; k < 2 * 256; k += kSweepThreads ) s_hist[k] = 0;
  if ( threadIdx.x < 2 * kKnots )
  {
    const int c = threadIdx.x / kKnots, q = threadIdx.x % kKnots, a = c ? axis2 : axis;
    const double from = pp->knot[a][q];
    const double per_unit = __ddiv_rn( static_cast< double >( kSteps ), __dsub_rn( pp->knot[a][q + 1], from ) );
    s_knot[c][q] = from;
    s_per[c][q] = per_unit;
    if ( blockIdx.x == 0 ) pw->cut[c][q] = make_double2( from, per_unit );  // for A's sweeps
  }
  if ( blockIdx.x == 0 && threadIdx.x == 0 )
  {
    pw->axis2 = axis2;
    pw->axis3 = 3 - axis - axis2;
  }
  __syncthreads();
  double w[2] = { 0.0, 0.0 };
  for ( uint64_t i = static_cast< uint64_t >( blockIdx.x ) * kSweepThreads + threadIdx.x; i < n;
        i += static_cast< uint64_t >( gridDim.x ) * kSweepThreads )
  {
    const double *src = verts + i * V * 3;
    uint32_t key = 0;
#pragma unroll
    for ( int c = 0; c < 2; ++c )
    {
      double lo, hi;
      cardinal_slab( src, V, c ? axis2 : axis, eps, lo, hi );
      key = ( key << 8 ) | strip_of( lo, s_knot[c], s_per[c] );
      const double x = __dsub_ru( hi, lo );
      w[c] = x > w[c] ? x : w[c];
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
      w[c] = x > w[c] ? x : w[c];
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
// Resident blocks: the compiler's own choice of registers spilled in the sweep's loop or left fewer warps (triangles at
// 18-DOP, 2 x 262,144: 338 us a call at 12 blocks, 290 at 8 to 9; hexahedra would get 3 blocks at 26-DOP).
template< int K, int VT >
constexpr int kSweepMinBlocks = K == 6 ? 12 : ( VT == 8 ? ( K == 26 ? 4 : 5 ) : ( K == 26 ? 8 : 9 ) );

template< int K, int VT >
__global__ void __launch_bounds__( kPairThreads, kSweepMinBlocks< K, VT > ) k_sweep(const double *__restrict__ verts, uint32_t Vrt, uint64_t na,
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
  const int axis = pp->axis, axis2 = pp->axis2, axis3 = pp->axis3;
  const unsigned lane = threadIdx.x & 31u, lt = ( 1u << lane ) - 1u;
  double( *rows )[K] = s_rows[threadIdx.x >> 5];
  const double2 *z = reinterpret_cast< const double2 * >( srows ) + static_cast< uint64_t >( axis3 ) * nb;
  const uint64_t first = static_cast< uint64_t >( ( blockIdx.x * kPairThreads + threadIdx.x ) >> 5 ) * per;
  uint32_t i = 0, span = 0;  // span: first strip, last strip, first bin, last bin
  const bool mine = lane < per && first + lane < na;
  if ( mine )
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
  }
  __syncwarp();  // the cuts are loaded here, not beside the vertices: their registers are free again
#pragma unroll
  for ( int c = 0; c < 2; ++c )
  {
    const double *slab = rows[lane] + 2 * ( c ? axis2 : axis );
    const double mn = mine ? slab[0] : 0.0, mx = mine ? slab[1] : 0.0;
    const double2 cut = __ldg( &pp->cut[c][lane] );
    const uint32_t s0 = strip_of( __dsub_rd( mn, ord_decode( pp->wmax_enc[c] ) ), cut.x, cut.y );
    span |= ( s0 | ( strip_of( mx, cut.x, cut.y ) << 8 ) ) << ( 16 * c );
  }
  __syncwarp();
  const uint32_t count = first < na ? static_cast< uint32_t >( min( static_cast< uint64_t >( per ), na - first ) ) : 0u;
  for ( uint32_t u = 0; u < count; ++u )
  {
    const uint32_t ai = __shfl_sync( 0xffffffffu, i, u ), sp = __shfl_sync( 0xffffffffu, span, u );
    const uint32_t s0 = sp & 255u, s1 = ( sp >> 8 ) & 255u, y0 = ( sp >> 16 ) & 255u, y1 = sp >> 24;
    const double *row = rows[u];
    const double zlo = row[2 * axis3], zhi = row[2 * axis3 + 1];
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
  // a quarter of the sample below 16,384 elements: the ranking of 256 ends before the axis beside it, that of 1,024 made a
  // call on 2 x 1,000 triangles 110 us instead of 101; from there on the more even strips are worth it (2 x 40,000: 147
  // instead of 149 us)
  const uint64_t want = x.na < ( 1u << 14 ) || x.nb < ( 1u << 14 ) ? kSample / 4 : kSample;
  const int cnt = static_cast< int >( x.nb < want ? x.nb : want ), per = ( cnt * kRankLanes + kSweepThreads - 1 ) / kSweepThreads;
  k_sweep_sample<<< 3 * per + ( axis < 0 ? kAxisBlocks : 0 ), kSweepThreads, 0, x.s >>>( x, axis, per, cnt,
                                                                                       static_cast< double >( x.nb ) / cnt );
  return cudaGetLastError();
}

cudaError_t launch_sweep_keys(const sweep_launch &x)
{
  const uint64_t blocks = ( x.nb + kSweepThreads - 1 ) / kSweepThreads, most = 2 * static_cast< uint64_t >( device_sm_count() );
  const unsigned grid = static_cast< unsigned >( blocks < most ? blocks : most );
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
