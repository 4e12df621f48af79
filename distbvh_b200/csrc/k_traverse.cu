// k_traverse.cu — tree traversal emitting candidate element pairs (K6), FP64 recheck (K7), gid output.
//
// The reference finds pairs with a 4-way simultaneous recursion over two trees (get_overlapping_indices,
// src/bvh/collision_query.hpp:293-329) or a per-entity descent (query_tree, collision_query.hpp:166-213), both
// pruning on the strict all-slab overlap (kdop.hpp:120-125, 538-549). Here a warp walks the other object's tree
// for a packet of 32 consecutive query ranks (Morton order: spatially coherent) by the packet's union box, filters the
// elements of the buckets that it reaches, and tests those against the packet's queries (see "the walk of one
// packet"). Overlaps are emitted as (query element, tree element) local indices through a per-warp buffer in shared
// memory; pairs beyond capacity are counted but not stored, so the host can grow the buffer and retry. In sparse
// contact the grid is persistent, culls 32 packets per warp step against the target root before walking the
// survivors, and computes the element slabs it tests; in dense contact it is one warp per packet, and the element
// slabs are stored. The FP64 recheck of the precision form reads both elements' vertices per candidate and decides
// the overlap by comparison-only projections (kdop_math.cuh).
//
// Self-collision (self_collision_set, collision_query.hpp:331-368): the query of rank i only visits subtrees
// holding ranks > i (internal node k splits its bucket range [l, r] into [l, k] and [k + 1, r]) and tests only
// bucket elements of rank > i, so every unordered pair is found once and no element is paired with itself.
#include <cstddef>

#include "bulk_copy.cuh"
#include "bvhg_internal.cuh"
#include "kdop_math.cuh"

namespace bvhg {
int device_sm_count();
namespace {

// Two warps per block: a block's shared memory is free for the next one when its slower walk ends (4 warps per block:
// the dense walks 4-5% slower).
constexpr int kTravThreads = 64;

// Resident blocks per SM of the walk that computes the element slabs it tests (128 registers).
constexpr int kTravBlocksPerSM = 4 * 128 / kTravThreads;

// Slabs of element e straight into a shared-memory row (K values: min, max per slab): the same FP64 slabs (slab by
// slab, so that only the vertices stay in registers), or the same FP32 enclosures, that slabs_body unites into the
// bucket boxes.
template< int K, typename T, int VT >
__device__ __forceinline__ void slabs_to_row(const double *__restrict__ verts, uint32_t Vrt, uint32_t e, double eps,
                                             float eps_hi, T *row)
{
  constexpr int D = K / 2;
  if constexpr ( VT > 0 && sizeof( T ) == 8 )
  {
    double p[VT * 3];
    const double *src = verts + static_cast< size_t >( e ) * VT * 3;
#pragma unroll
    for ( int k = 0; k < VT * 3; ++k ) p[k] = __ldg( src + k );
#pragma unroll
    for ( int a = 0; a < D; ++a )
    {
      double l, h;
      slab64< K >( p, VT, a, eps, l, h );
      row[2 * a] = l;
      row[2 * a + 1] = h;
    }
  } else {
    T lo[D], hi[D];
    leaf_slabs< K, T, VT >( verts, Vrt, e, eps, eps_hi, lo, hi );
#pragma unroll
    for ( int a = 0; a < D; ++a )
    {
      row[2 * a] = lo[a];
      row[2 * a + 1] = hi[a];
    }
  }
}

// The three cardinal slabs of element e, as leaf_slabs forms them.
template< int K, typename T, int VT >
__device__ __forceinline__ void cardinal_slabs(const double *__restrict__ verts, uint32_t Vrt, uint32_t e, double eps,
                                               float eps_hi, T *lo, T *hi)
{
  leaf_slabs< 6, T, VT >( verts, Vrt, e, eps, eps_hi, lo, hi );
}

// Everything one query packet needs besides the tree (see walk_packet).
template< typename T >
struct trav_args
{
  const T *qwarp;
  const double *qverts;
  uint32_t qV;
  const T *qrows;    // query element slabs in rank order (stored form only)
  const uint32_t *qperm;
  uint32_t nq;
  const int2 *child;
  const T *nbox;
  const int2 *range;
  const double *tverts;
  uint32_t tV;
  const T *tcache;   // element slabs of the target in rank order (stored form only)
  const uint32_t *tperm;
  const obj_scalars *tsc;
  uint32_t nt;
  int self;
  double eps;
  float eps_hi;
  uint2 *pairs;
  uint64_t cap;
  pair_scalars *ps;
  int stack_limit;  // stack bound of the walk over stored slabs (kWalkStack, lower under a test hook)
};

// The typed view of a scene's traversal item.
template< typename T >
__device__ __forceinline__ trav_args< T > typed(const trav_item &it)
{
  trav_args< T > x;
  x.qwarp = static_cast< const T * >( it.qwarp );
  x.qverts = it.qverts;
  x.qV = it.qV;
  x.qrows = static_cast< const T * >( it.qrows );
  x.qperm = it.qperm;
  x.nq = it.nq;
  x.child = it.child;
  x.nbox = static_cast< const T * >( it.nbox );
  x.range = it.range;
  x.tverts = it.tverts;
  x.tV = it.tV;
  x.tcache = static_cast< const T * >( it.tcache );
  x.tperm = it.tperm;
  x.tsc = it.tsc;
  x.nt = it.nt;
  x.self = it.self;
  x.eps = it.eps;
  x.eps_hi = it.eps_hi;
  x.pairs = it.pairs;
  x.cap = it.cap;
  x.ps = it.ps;
  x.stack_limit = it.dense_stack;
  return x;
}

// ---- the walk of one packet -----------------------------------------------------------------------------------
//
// A packet is 32 consecutive query ranks and belongs to one warp. Its walk has five kinds of steps, each with its own
// use of the lanes:
//   - Expand: lane = (node, child). Up to 16 nodes are popped from the packet's stack; every lane tests one child's
//     slabs against the packet's union box. A leaf bucket that passes goes onto the bucket list, an internal node back
//     onto the stack; children smaller than half the packet's box go onto the check list first.
//   - Check: lane = query. The cardinal slabs of the listed boxes are staged in shared memory, eight boxes at a time
//     with the next eight on their way, and every lane tests its query against them. A child that no query overlaps is
//     dropped, and a bucket is listed with the queries that overlap it.
//   - Filter: lane = element of four listed buckets. The elements that overlap the packet's union box are gathered, 16
//     at a time, as rows in shared memory, and with them the queries of their buckets.
//   - Cardinal tests: lane = (query of two, gathered element), the element's cardinal slabs in registers, over those
//     queries. Survivors collect in a list in shared memory.
//   - Slab tests: lane = survivor (query, element), on the other slabs.
// Everything larger than a query costs one lane-test per box or element instead of 32. On a tet lattice at 26-DOP a
// packet meets 157 nodes, 49 buckets of 390 elements, 149 elements that overlap its box, 310 survivors and 133 pairs
// (counted on the host over 64^3 cells). A walk of (node, lane mask) entries that tests all 32 queries against every
// node, and every query against every element of the buckets that it overlaps, makes 175 x 64 box tests and 1455
// element tests on all slabs for them, most on idle lanes.
// What bounds it is the chain of dependent reads and the instructions per test, so a step reads all slabs of its nodes
// or elements at once (one trip to memory per step) and compares without branches.
// Traversal of the 256^3 lattice at 26-DOP FP64 25.6 -> 12.3 ms; 161^3 at 18-DOP FP32 2.53 -> 1.30 ms; 200,003
// tetrahedra against themselves 208 -> 128 us; two plates of 10,000 triangles 186 -> 91 us (52 in narrow packets); in
// sparse contact the sphere on the plate (9.4M triangles) 105 -> 59 us. Measured and slower: the same expansion, then all
// 32 queries against every bucket and four queries by eight elements per round from shared memory (15.4 ms); the same
// with a second round for the non-cardinal slabs by (survivor, slab) lanes (29 ms); rows read five slabs at a time (20 to
// 50 ms, depending on the resident warps).
// A packet whose ranks straddle a jump of the Morton curve, or whose elements lie far apart, or one of whose elements is
// long, has a union box that says little: the check of the small children keeps its walk on the nodes that one of its
// queries overlaps, and the buckets' queries keep the cardinal tests on those. (Testing all queries of the packet against
// every gathered element: 300,000 triangles of which 100 span half the domain against 300,000 small ones 15.1 ms instead
// of 8.65, one in 1,000 spanning 0.3 of it 2.8 instead of 1.62 ms, and the even lattices 13.9 and 1.46 instead of 12.9
// and 1.33 ms. Waiting for every eight boxes of a check: 8.65, 1.62, 12.9 and 1.33 ms instead of 8.47, 1.55, 12.3 and
// 1.30.)
//
// The element slabs come from the rows that the slab kernel stored (STORED: dense contact; slab-major per bucket, so
// that the filter reads the pairs of one slab of eight elements as one piece) or are computed from the vertices: the
// packet's 32 queries once, and the gathered elements (there the filter tests the cardinal slabs only).
//
// Stack bound: the wide steps stop while stack and list hold more than stack_limit - 32 - kWalkDepth entries; the walk
// then expands one node at a time and checks the list after each, which is a depth-first walk and adds at most one
// entry per tree level (at most 95). kWalkStack entries therefore always suffice. A lower stack_limit (test hook) can
// be reached: the walk raises kErrOverflowStack, and the host runs the pair search again with computed slabs.
constexpr int kWalkDepth = 96;  // radix tree over 96-bit (key, rank) pairs: at most 95 internal levels
constexpr int kWalkStack = 284;
constexpr int kCheckCap = 64;   // listed children: checked once more than 32 are held
constexpr int kCheckRows = 8;   // boxes staged per check step
constexpr int kLeafCap = 64;    // listed buckets: filtered once more than 32 are held
constexpr int kGather = 16;     // elements gathered before they are tested
constexpr int kSurvivors = 96;  // (query, element) pairs past the cardinal tests: tested once 32 are held
constexpr int kPairBuf = 64;    // buffered pairs per warp: drained once more than 32 are held

template< int K, typename T >
struct walk_smem
{
  // read as (min, max) pairs, and written by asynchronous copies of pairs
  alignas( 16 ) T q[32][K];             // slabs of the packet's queries
  alignas( 16 ) T e[kGather][K];        // slabs of the gathered elements
  alignas( 16 ) T rows[2][kCheckRows][6];  // cardinal slabs of the boxes being checked and of the next ones
  alignas( 16 ) T g[K];                 // the packet's union box
  alignas( 16 ) uint2 out[kPairBuf];    // pairs found and not yet written
  int list[kCheckCap];                  // children to check: 2 * parent + side
  int leaf[kLeafCap];                   // buckets to filter
  unsigned mask[kLeafCap];              // the queries that may overlap each of them
  int stack[kWalkStack];                // internal nodes to expand
  uint32_t qe[32];                      // query element indices
  uint32_t te[kGather], tr[kGather];    // element indices and ranks of the gathered elements
  uint16_t surv[kSurvivors];            // query | gathered element << 8
};

// The state of a warp's walk.
struct walk_state
{
  uint32_t i0;    // first query rank of the packet
  unsigned lane;
  unsigned in;    // queries that overlap the target's root box
  int ne = 0;     // gathered elements
  unsigned any = 0;  // queries that may overlap one of them
  uint32_t ns = 0, nout = 0;
};

// A (min, max) pair: from global memory (read-only path) or from shared memory, as one vector load.
__device__ __forceinline__ void load_pair(const double *p, double &lo, double &hi)
{
  const double2 v = __ldg( reinterpret_cast< const double2 * >( p ) );
  lo = v.x;
  hi = v.y;
}
__device__ __forceinline__ void load_pair(const float *p, float &lo, float &hi)
{
  const float2 v = __ldg( reinterpret_cast< const float2 * >( p ) );
  lo = v.x;
  hi = v.y;
}
__device__ __forceinline__ void shared_pair(const double *p, double &lo, double &hi)
{
  const double2 v = *reinterpret_cast< const double2 * >( p );
  lo = v.x;
  hi = v.y;
}
__device__ __forceinline__ void shared_pair(const float *p, float &lo, float &hi)
{
  const float2 v = *reinterpret_cast< const float2 * >( p );
  lo = v.x;
  hi = v.y;
}
__device__ __forceinline__ void copy_pair(double *dst, const double *src) { cp_async16( dst, src ); }
__device__ __forceinline__ void copy_pair(float *dst, const float *src) { cp_async_small< 8 >( dst, src ); }

// Writes the warp's buffered pairs: one atomic reservation for all of them, then coalesced stores (a count past
// the capacity is still counted, so the host learns the size it needs).
template< int K, typename T >
__device__ __forceinline__ void drain_pairs(const trav_args< T > &x, walk_smem< K, T > &sm, walk_state &w)
{
  __syncwarp();
  unsigned long long base = 0;
  if ( w.lane == 0 && w.nout ) base = atomicAdd( &x.ps->count, static_cast< unsigned long long >( w.nout ) );
  base = __shfl_sync( 0xffffffffu, base, 0 );
  for ( uint32_t j = w.lane; j < w.nout; j += 32 )
    if ( base + j < x.cap ) x.pairs[base + j] = sm.out[j];
  __syncwarp();
  w.nout = 0;
}

// Appends the pairs (q, e) of the lanes with hit.
template< int K, typename T >
__device__ __forceinline__ void emit(const trav_args< T > &x, walk_smem< K, T > &sm, walk_state &w, bool hit, uint32_t q, uint32_t e)
{
  const unsigned m = __ballot_sync( 0xffffffffu, hit );
  if ( !m ) return;
  if ( hit ) sm.out[w.nout + __popc( m & ( ( 1u << w.lane ) - 1u ) )] = make_uint2( sm.qe[q], sm.te[e] );
  w.nout += static_cast< uint32_t >( __popc( m ) );
  if ( w.nout > kPairBuf - 32 ) drain_pairs( x, sm, w );
}

// The slab tests of `count` (at most 32) listed survivors from `first` on.
template< int K, typename T >
__device__ __forceinline__ void test_survivors(const trav_args< T > &x, walk_smem< K, T > &sm, walk_state &w, uint32_t first,
                                               uint32_t count)
{
  constexpr int D = K / 2;
  const bool act = w.lane < count;
  const uint32_t s = act ? sm.surv[first + w.lane] : 0u, q = s & 31u, e = s >> 8;
  const T *qr = sm.q[q], *er = sm.e[e];
  bool lo_ok = act, hi_ok = true;  // bitwise: no branch per comparison
#pragma unroll
  for ( int a = 3; a < D; ++a )
  {
    T ql, qh, el, eh;
    shared_pair( qr + 2 * a, ql, qh );
    shared_pair( er + 2 * a, el, eh );
    lo_ok &= ql < eh;
    hi_ok &= el < qh;
  }
  emit( x, sm, w, lo_ok & hi_ok, q, e );
}

// All tests of the gathered elements; leaves none. Half a warp takes one query each round (two rounds in flight).
template< int K, typename T >
__device__ __forceinline__ void test_gathered(const trav_args< T > &x, walk_smem< K, T > &sm, walk_state &w)
{
  cp_async_wait_all();
  __syncwarp();
  const uint32_t e = w.lane & ( kGather - 1u );
  const bool act = static_cast< int >( e ) < w.ne, upper = w.lane >= kGather;
  T el[3], eh[3];
#pragma unroll
  for ( int a = 0; a < 3; ++a ) shared_pair( &sm.e[e][2 * a], el[a], eh[a] );
  // self-collision: only the queries of lower rank
  const uint32_t above = act ? ( x.self ? sm.tr[e] - w.i0 : 32u ) : 0u;
  constexpr int U = 2;
  for ( unsigned m = w.any; m; )
  {
    uint32_t q[U];
    bool ok[U];
#pragma unroll
    for ( int u = 0; u < U; ++u )
    {
      const unsigned rest = m & ( m - 1u );
      const unsigned mine = upper ? rest : m;
      ok[u] = mine != 0u;
      q[u] = mine ? static_cast< uint32_t >( __ffs( mine ) - 1 ) : 0u;
      m = rest & ( rest - 1u );
      ok[u] &= q[u] < above;
      const T *qr = sm.q[q[u]];
#pragma unroll
      for ( int a = 0; a < 3; ++a )
      {
        T ql, qh;
        shared_pair( qr + 2 * a, ql, qh );
        ok[u] &= ( ql < eh[a] ) & ( el[a] < qh );
      }
    }
#pragma unroll
    for ( int u = 0; u < U; ++u )
    {
      if constexpr ( K == 6 )
      {
        emit( x, sm, w, ok[u], q[u], e );
      } else {
        const unsigned bal = __ballot_sync( 0xffffffffu, ok[u] );
        if ( ok[u] ) sm.surv[w.ns + __popc( bal & ( ( 1u << w.lane ) - 1u ) )] = static_cast< uint16_t >( q[u] | ( e << 8 ) );
        w.ns += static_cast< uint32_t >( __popc( bal ) );
      }
    }
    if constexpr ( K > 6 )
    {
      if ( w.ns >= 32u )
      {
        // the last 32 (or twice 32) are tested; the others stay where they are
        __syncwarp();
        do
        {
          w.ns -= 32u;
          test_survivors( x, sm, w, w.ns, 32u );
        } while ( w.ns >= 32u );
        __syncwarp();
      }
    }
  }
  if constexpr ( K > 6 )
  {
    if ( w.ns )
    {
      __syncwarp();
      test_survivors( x, sm, w, 0u, w.ns );
      w.ns = 0;
    }
  }
  __syncwarp();
  w.ne = 0;
  w.any = 0;
}

// The filter of the nleaf listed buckets.
template< int K, typename T, int VT, bool STORED >
__device__ __forceinline__ void filter_buckets(const trav_args< T > &x, walk_smem< K, T > &sm, walk_state &w, int nleaf)
{
  constexpr int D = K / 2;
  for ( int b0 = 0; b0 < nleaf; b0 += 4 )
  {
    const int b = b0 + static_cast< int >( w.lane >> 3 );
    const int bucket = b < nleaf ? sm.leaf[b] : 0;
    const uint32_t r = static_cast< uint32_t >( kLeafSize * bucket ) + ( w.lane & 7u );
    bool o = b < nleaf && r < x.nt && ( !x.self || r > w.i0 );
    const uint32_t te = o ? __ldg( x.tperm + r ) : 0u;
    const T *src = STORED ? x.tcache + static_cast< size_t >( bucket ) * ( kLeafSize * K ) + 2 * ( w.lane & 7u ) : nullptr;
    bool lo_ok = true, hi_ok = true;  // bitwise: no branch per comparison
    if ( o )
    {
      // all slabs at once (stored form): one trip to memory per four buckets
      constexpr int F = STORED ? D : 3;
      T lo[F], hi[F];
      if constexpr ( STORED )
      {
#pragma unroll
        for ( int a = 0; a < F; ++a ) load_pair( src + 2 * kLeafSize * a, lo[a], hi[a] );
      } else {
        cardinal_slabs< K, T, VT >( x.tverts, x.tV, te, x.eps, x.eps_hi, lo, hi );
      }
#pragma unroll
      for ( int a = 0; a < F; ++a )
      {
        T gl, gh;
        shared_pair( &sm.g[2 * a], gl, gh );
        lo_ok &= gl < hi[a];
        hi_ok &= lo[a] < gh;
      }
      o = lo_ok & hi_ok;
    }
    // the elements that passed become rows; full rows are tested
    for ( unsigned m = __ballot_sync( 0xffffffffu, o ); m; )
    {
      const int at = w.ne + __popc( m & ( ( 1u << w.lane ) - 1u ) );
      const bool put = ( ( m >> w.lane ) & 1u ) && at < kGather;
      if ( put )
      {
        sm.te[at] = te;
        sm.tr[at] = r;
        if constexpr ( STORED )
        {
#pragma unroll
          for ( int a = 0; a < D; ++a ) copy_pair( &sm.e[at][2 * a], src + 2 * kLeafSize * a );
        } else {
          slabs_to_row< K, T, VT >( x.tverts, x.tV, te, x.eps, x.eps_hi, sm.e[at] );
        }
      }
      w.ne = min( kGather, w.ne + __popc( m ) );
      w.any |= __reduce_or_sync( 0xffffffffu, put ? sm.mask[b] : 0u );
      m &= ~__ballot_sync( 0xffffffffu, put );
      if ( w.ne == kGather ) test_gathered( x, sm, w );
    }
  }
  __syncwarp();
}

// One packet: ranks i0 .. i0 + width - 1 (width 8 or 32) against the target tree (see above). rb: the target root's
// slabs.
template< int K, typename T, int VT, bool STORED >
__device__ __forceinline__ void walk_packet(const trav_args< T > &x, const uint32_t i0, const uint32_t width,
                                            const unsigned lane, walk_smem< K, T > &sm, const T *rb)
{
  constexpr int D = K / 2;
  const uint32_t i = i0 + lane;
  const T *wb = x.qwarp + static_cast< size_t >( i0 >> 5 ) * K;
  // 1. The union box of the 32 ranks around the packet against the target's root box (uniform over the warp).
  {
    bool o = true;
#pragma unroll
    for ( int a = 0; a < D; ++a ) o = o && ( __ldg( wb + 2 * a ) < rb[2 * a + 1] && rb[2 * a] < __ldg( wb + 2 * a + 1 ) );
    if ( !o ) return;
  }
  // 2. Each lane's own slabs (stored, or from its element's vertices) against the root box.
  const bool valid = i < x.nq && lane < width;
  const uint32_t qe = valid ? __ldg( x.qperm + i ) : 0u;
  if constexpr ( STORED )
  {
    const uint32_t iv = valid ? i : i0;
    const T *qs = x.qrows + static_cast< size_t >( iv >> 3 ) * ( kLeafSize * K ) + 2 * ( iv & 7u );
#pragma unroll
    for ( int a = 0; a < D; ++a ) copy_pair( &sm.q[lane][2 * a], qs + 2 * kLeafSize * a );
    cp_async_wait_all();
  } else {
    if ( valid ) slabs_to_row< K, T, VT >( x.qverts, x.qV, qe, x.eps, x.eps_hi, sm.q[lane] );
  }
  sm.qe[lane] = qe;
  __syncwarp();
  bool in_root = valid;
#pragma unroll
  for ( int a = 0; a < D; ++a )
  {
    T ql, qh;
    shared_pair( &sm.q[lane][2 * a], ql, qh );
    in_root = in_root && ( ql < rb[2 * a + 1] && rb[2 * a] < qh );
  }
  walk_state w;
  w.i0 = i0;
  w.lane = lane;
  w.in = __ballot_sync( 0xffffffffu, in_root );
  if ( !w.in ) return;
  // 3. The packet's union box: the group's, or that of the narrow packet's queries which overlap the root (their slabs
  // are numbers; a NaN of another query must not reach the box).
  if ( width == 32u )
  {
    if ( lane < K ) sm.g[lane] = __ldg( wb + lane );
  } else if ( lane < D ) {
    unsigned m = w.in;
    T lo, hi;
    shared_pair( &sm.q[__ffs( m ) - 1][2 * lane], lo, hi );
    while ( m &= m - 1u )
    {
      T l, h;
      shared_pair( &sm.q[__ffs( m ) - 1][2 * lane], l, h );
      lo = l < lo ? l : lo;
      hi = hi < h ? h : hi;
    }
    sm.g[2 * lane] = lo;
    sm.g[2 * lane + 1] = hi;
  }
  __syncwarp();
  const int root = x.tsc->root;
  const unsigned lt = ( 1u << lane ) - 1u;
  const int limit = STORED ? x.stack_limit : kWalkStack;
  int sp = 0, nl = 0, nleaf = 0;
  bool full = false;  // the stack bound was reached (uniform over the warp)
  if ( lane == 0 )
  {
    sm.mask[0] = w.in;
    if ( root < 0 ) sm.leaf[0] = ~root;
    else sm.stack[0] = root;
  }
  if ( root < 0 ) nleaf = 1;
  else sp = 1;
  const T half = T( 0.5 ) * ( ( sm.g[1] - sm.g[0] ) + ( sm.g[3] - sm.g[2] ) + ( sm.g[5] - sm.g[4] ) );
  while ( !full && ( sp > 0 || nl > 0 ) )
  {
    __syncwarp();
    if ( nleaf > kLeafCap - 32 )
    {
      filter_buckets< K, T, VT, STORED >( x, sm, w, nleaf );
      nleaf = 0;
    }
    const bool wide = sp + nl + 32 + kWalkDepth <= limit;
    if ( sp > 0 && nl <= kCheckCap - 32 && ( wide || nl == 0 ) )
    {
      // expand: lane = (node, child), the child against the packet's union box
      const int p = wide ? min( sp, 16 ) : 1;
      const int k = static_cast< int >( lane >> 1 ), side = static_cast< int >( lane & 1u );
      bool o = k < p;
      const int node = o ? sm.stack[sp - 1 - k] : 0;
      sp -= p;
      int c = 0;
      bool small = false;
      if ( o )
      {
        c = __ldg( reinterpret_cast< const int * >( x.child ) + 2 * node + side );
        const T *nb = x.nbox + static_cast< size_t >( node ) * D * 4 + 2 * side;
        T lo[D], hi[D];
#pragma unroll
        for ( int a = 0; a < D; ++a ) load_pair( nb + a * 4, lo[a], hi[a] );
        if ( x.self )
        {
          // left child covers buckets [l, node], right child [node + 1, r]: skip subtrees whose last rank <= i0
          const int last = side ? __ldg( &x.range[node].y ) : node;
          o = min( kLeafSize * last + kLeafSize - 1, static_cast< int >( x.nt ) - 1 ) > static_cast< int >( i0 );
        }
        small = ( hi[0] - lo[0] ) + ( hi[1] - lo[1] ) + ( hi[2] - lo[2] ) < half;
        bool lo_ok = true, hi_ok = true;  // bitwise: no branch per comparison
#pragma unroll
        for ( int a = 0; a < D; ++a )
        {
          T gl, gh;
          shared_pair( &sm.g[2 * a], gl, gh );
          lo_ok &= gl < hi[a];
          hi_ok &= lo[a] < gh;
        }
        o = o & lo_ok & hi_ok;
      }
      const unsigned ml = __ballot_sync( 0xffffffffu, o && small );
      const unsigned mp = __ballot_sync( 0xffffffffu, o && !small && c >= 0 );
      const unsigned mb = __ballot_sync( 0xffffffffu, o && !small && c < 0 );
      full = sp + __popc( mp ) > limit;
      if ( full ) break;
      if ( o )
      {
        if ( small ) sm.list[nl + __popc( ml & lt )] = 2 * node + side;
        else if ( c >= 0 ) sm.stack[sp + __popc( mp & lt )] = c;
        else
        {
          sm.leaf[nleaf + __popc( mb & lt )] = ~c;
          sm.mask[nleaf + __popc( mb & lt )] = w.in;
        }
      }
      nl += __popc( ml );
      sp += __popc( mp );
      nleaf += __popc( mb );
      continue;
    }
    // check: lane = query, the listed boxes' cardinal slabs against every query of the packet; the next boxes are on their
    // way meanwhile
    int link = 0, next_link = 0;  // of the child whose slab this lane copies
    auto stage = [&](int b0, int buf) {
      static_assert( kCheckRows * 3 <= 32, "one pair per lane" );
      const int k = static_cast< int >( lane ) / 3, a = static_cast< int >( lane ) - 3 * k;
      if ( k < min( kCheckRows, nl - b0 ) )
      {
        const int e = sm.list[b0 + k];
        copy_pair( &sm.rows[buf][k][2 * a], x.nbox + static_cast< size_t >( e >> 1 ) * D * 4 + a * 4 + ( e & 1 ) * 2 );
        next_link = __ldg( reinterpret_cast< const int * >( x.child ) + e );
      }
      cp_async_commit();
    };
    stage( 0, 0 );
    for ( int b0 = 0, buf = 0; b0 < nl && !full; b0 += kCheckRows, buf ^= 1 )
    {
      const int nb = min( kCheckRows, nl - b0 );
      link = next_link;
      stage( b0 + kCheckRows, buf ^ 1 );
      cp_async_wait_older();
      __syncwarp();
      unsigned alive = in_root ? ( 1u << nb ) - 1u : 0u;
#pragma unroll
      for ( int a = 0; a < 3; ++a )
      {
        T ql, qh;
        shared_pair( &sm.q[lane][2 * a], ql, qh );
#pragma unroll
        for ( int j = 0; j < kCheckRows; ++j )
        {
          T bl, bh;
          shared_pair( &sm.rows[buf][j][2 * a], bl, bh );
          const bool o = ( ql < bh ) & ( bl < qh );
          alive &= o ? ~0u : ~( 1u << j );
        }
      }
      for ( int j = 0; j < nb; ++j )
      {
        const unsigned who = __ballot_sync( 0xffffffffu, ( alive >> j ) & 1u );  // the queries that overlap box j
        if ( !who ) continue;
        const int ch = __shfl_sync( 0xffffffffu, link, 3 * j );
        if ( ch < 0 )
        {
          if ( nleaf == kLeafCap )
          {
            __syncwarp();
            filter_buckets< K, T, VT, STORED >( x, sm, w, nleaf );
            nleaf = 0;
          }
          if ( lane == 0 )
          {
            sm.leaf[nleaf] = ~ch;
            sm.mask[nleaf] = who;
          }
          ++nleaf;
        } else if ( sp < limit ) {
          if ( lane == 0 ) sm.stack[sp] = ch;
          ++sp;
        } else {
          full = true;
        }
      }
      __syncwarp();  // the rows are refilled by the next boxes
    }
    nl = 0;
  }
  __syncwarp();
  filter_buckets< K, T, VT, STORED >( x, sm, w, nleaf );
  if ( w.ne ) test_gathered( x, sm, w );
  if ( full && lane == 0 ) atomicCAS( &x.ps->error, 0, kErrOverflowStack );
  drain_pairs( x, sm, w );
}

// Roots first: objects far apart (most pairs of a batch) end here for the whole grid. No tree exists after a failed
// sort of either object.
template< int K, typename T >
__device__ __forceinline__ bool objects_meet(const trav_args< T > &x, const obj_scalars *__restrict__ qsc)
{
  if ( *reinterpret_cast< const volatile int * >( &x.tsc->error ) == kErrTimeout ||
       *reinterpret_cast< const volatile int * >( &qsc->error ) == kErrTimeout )
    return false;
  constexpr int D0 = K / 2 < 4 ? K / 2 : 4;
  const T *rb = reinterpret_cast< const T * >( x.tsc->root_box );
  const T *qr = reinterpret_cast< const T * >( qsc->root_box );
  bool o = true;
#pragma unroll
  for ( int a = 0; a < D0; ++a ) o = o && ( qr[2 * a] < rb[2 * a + 1] && rb[2 * a] < qr[2 * a + 1] );
  return o;
}

// Sparse contact: a persistent grid. A warp takes chunks from the pair counters' packet dispenser; chunk c holds the
// packets c, c + C, c + 2C, ... (C chunks, at most 32 packets each), so a contact region (consecutive Morton ranks) is
// spread over many chunks. Lane j tests the union box of the chunk's packet j against the target root (one load per
// lane for the packets far from the target), then the warp walks the survivors one after the other.
template< int K, typename T, int VT >
__device__ void traverse_body(const trav_item &item, uint32_t, uint32_t)
{
  const trav_args< T > x = typed< T >( item );
  constexpr int D = K / 2;
  extern __shared__ __align__( 16 ) unsigned char s_walk[];
  auto &sm = reinterpret_cast< walk_smem< K, T > * >( s_walk )[threadIdx.x >> 5];
  const unsigned lane = threadIdx.x & 31u;
  if ( !objects_meet< K, T >( x, item.qsc ) ) return;
  const T *rb = reinterpret_cast< const T * >( x.tsc->root_box );
  const uint32_t packets = ( x.nq + 31 ) / 32;
  const uint32_t chunks = ( packets + item.chunk - 1 ) / item.chunk;
  while ( true )
  {
    uint32_t c = 0;
    if ( lane == 0 ) c = atomicAdd( &x.ps->packet_next, 1u );
    c = __shfl_sync( 0xffffffffu, c, 0 );
    if ( c >= chunks ) break;
    const uint64_t pk = c + static_cast< uint64_t >( lane ) * chunks;
    bool o = false;
    if ( lane < item.chunk && pk < packets )
    {
      const T *wb = x.qwarp + pk * D * 2;
      o = true;
#pragma unroll
      for ( int a = 0; a < D; ++a ) o = o && ( __ldg( wb + 2 * a ) < rb[2 * a + 1] && rb[2 * a] < __ldg( wb + 2 * a + 1 ) );
    }
    for ( unsigned m = __ballot_sync( 0xffffffffu, o ); m; m &= m - 1 )
    {
      const uint32_t p = c + static_cast< uint32_t >( __ffs( m ) - 1 ) * chunks;
      walk_packet< K, T, VT, false >( x, p * 32, 32u, lane, sm, rb );
    }
  }
}

// Dense contact: one warp per packet (the hardware balances the walks).
template< int K, typename T >
__device__ void stored_body(const trav_item &item, uint32_t bid, uint32_t)
{
  const trav_args< T > x = typed< T >( item );
  extern __shared__ __align__( 16 ) unsigned char s_walk[];
  auto &sm = reinterpret_cast< walk_smem< K, T > * >( s_walk )[threadIdx.x >> 5];
  const unsigned lane = threadIdx.x & 31u;
  if ( !objects_meet< K, T >( x, item.qsc ) ) return;
  const T *rb = reinterpret_cast< const T * >( x.tsc->root_box );
  const uint32_t width = item.width;
  const uint32_t pk = ( bid * blockDim.x + threadIdx.x ) >> 5;
  if ( static_cast< uint64_t >( pk ) * width < x.nq ) walk_packet< K, T, 0, true >( x, pk * width, width, lane, sm, rb );
}

// Shared memory per block of the walks, and their resident blocks per SM: as many as it allows (228 KB per SM, 1 KB of
// it reserved per block) up to a cap on the registers. Most forms compile without spills at it; a few bytes are spilled
// by the stored walks at 26-DOP and 18-DOP FP32 and by triangles at 26-DOP FP64 in sparse contact, and hexahedra in
// sparse contact, whose slabs are formed from 24 coordinates in registers, spill 234 bytes at 26-DOP FP64 and 110 at
// 18-DOP.
template< int K, typename T, bool STORED >
constexpr int kWalkSmem = ( kTravThreads / 32 ) * static_cast< int >( sizeof( walk_smem< K, T > ) );
template< int K, typename T, bool STORED >
constexpr int kWalkBySmem = ( 228 * 1024 ) / ( kWalkSmem< K, T, STORED > + 1024 );
template< int K, typename T, bool STORED >
constexpr int kWalkCap = STORED ? ( sizeof( T ) == 4 ? 8 : 6 ) * 128 / kTravThreads : kTravBlocksPerSM;
template< int K, typename T, bool STORED >
constexpr int kWalkBlocks = kWalkBySmem< K, T, STORED > < kWalkCap< K, T, STORED > ? kWalkBySmem< K, T, STORED >
                                                                                  : kWalkCap< K, T, STORED >;

// One scene's item and grid. Dense contact: one warp per packet. Sparse: a persistent grid of at most the resident
// blocks (8 per SM), whose warps take chunks of 1 to 32 packets.
//
// Queries per packet in dense contact. A walk is a chain of steps: a small object whose packets of 32 do not fill the
// device takes packets of one bucket (8), four times the warps with shorter chains. The line is where the narrow packets
// fill the 16 warps per SM of the form with the fewest resident ones (26-DOP FP64; kWalkBlocks gives the others 20 to
// 32), one line for all forms, found by measuring on both sides of it at 18- and 26-DOP FP64: two plates of 1,600 / 10,000
// triangles 64 / 91 -> 33 / 59 us, two blocks of 512 / 8,000 hexahedra 39 / 100 -> 22 / 54 us; beyond it the work of the
// narrow packets counts: 32,768 hexahedra 53 -> 64 us, 70,000 tetrahedra against themselves 83 -> 113 us, and a batch,
// whose scenes share the device, 9.8 -> 13.3 ms.
constexpr uint64_t kNarrowQueries = 148 * 16 * 8;

template< int K, typename T >
void trav_item_t(tree_view q, tree_view t, bool self, bool dense, bool alone, double eps, uint2 *pairs, uint64_t cap,
                 pair_scalars *ps, int dense_stack_limit, trav_item *it, uint32_t *blocks, bool *dense_out)
{
  it->qwarp = q.warp_box;
  it->qverts = q.verts;
  it->qV = q.V;
  it->qrows = q.elem_cache;
  it->qperm = q.perm;
  it->nq = static_cast< uint32_t >( q.n );
  it->child = t.child;
  it->nbox = t.node_box;
  it->range = t.range;
  it->tverts = t.verts;
  it->tV = t.V;
  it->tcache = t.elem_cache;
  it->tperm = t.perm;
  it->tsc = t.sc;
  it->nt = static_cast< uint32_t >( t.n );
  it->self = self ? 1 : 0;
  it->eps = eps;
  it->eps_hi = f32_round_up( eps );
  it->pairs = pairs;
  it->cap = cap;
  it->ps = ps;
  it->dense_stack = dense_stack_limit > 0 && dense_stack_limit < kWalkStack ? dense_stack_limit : kWalkStack;
  it->qsc = q.sc;
  constexpr uint64_t kWarps = kTravThreads / 32;
  // Packets per chunk in sparse contact: the survivors of a chunk are walked one after the other, so a small object
  // takes chunks of fewer packets, down to one, until there are two per resident warp. Traversal of spheres of 327,680
  // and 1.3M triangles on plates 60 -> 45 us (26-DOP FP64) and 55 -> 38 us (18-DOP FP32). Scenes of a batch, which share the device, keep 32.
  const uint64_t packets = ( q.n + 31 ) / 32;
  const uint64_t resident = static_cast< uint64_t >( device_sm_count() ) * kTravBlocksPerSM;
  const uint64_t per = packets / ( 2 * resident * kWarps );
  it->chunk = alone && per < 32 ? static_cast< uint32_t >( per ? per : 1 ) : 32u;
  const uint64_t chunks = ( packets + it->chunk - 1 ) / it->chunk;
  dense = dense && q.stored && t.stored;
  it->width = alone && q.n <= kNarrowQueries ? 8u : 32u;
  const uint64_t width = it->width;
  uint64_t b = dense ? ( ( q.n + width - 1 ) / width + kWarps - 1 ) / kWarps : ( chunks + kWarps - 1 ) / kWarps;
  if ( !dense && b > resident ) b = resident;
  *blocks = static_cast< uint32_t >( b < ( 1ull << 30 ) ? ( b ? b : 1 ) : ( 1ull << 30 ) );
  *dense_out = dense;
}

// A walk's two launch forms.
template< int K, typename T, int VT, bool STORED >
struct walk_kernels
{
  static constexpr int MB = kWalkBlocks< K, T, STORED >;
  static constexpr int smem = kWalkSmem< K, T, STORED >;
  static_assert( smem <= 48 * 1024, "more shared memory per block needs the opt-in" );
  static constexpr auto single()
  {
    if constexpr ( STORED ) return &k_single< trav_item, stored_body< K, T >, kTravThreads, MB >;
    else return &k_single< trav_item, traverse_body< K, T, VT >, kTravThreads, MB >;
  }
  static constexpr auto batched()
  {
    if constexpr ( STORED ) return &k_batched< trav_item, stored_body< K, T >, kTravThreads, MB >;
    else return &k_batched< trav_item, traverse_body< K, T, VT >, kTravThreads, MB >;
  }
  static cudaError_t launch(const trav_item &it, uint32_t grid, cudaStream_t s)
  {
    single()<<< grid, kTravThreads, smem, s >>>( it );
    return cudaGetLastError();
  }
  static cudaError_t launch_batch(const batch_launch &b, cudaStream_t s)
  {
    batched()<<< b.blocks, kTravThreads, smem, s >>>( static_cast< const trav_item * >( b.items ), b.starts, b.nitems );
    return cudaGetLastError();
  }
};

template< int K, typename T >
cudaError_t launch_trav_t(tree_view q, tree_view t, bool self, bool dense, double eps, uint2 *pairs, uint64_t cap,
                          pair_scalars *ps, cudaStream_t s, int dense_stack_limit, bool alone)
{
  trav_item it;
  uint32_t grid = 0;
  trav_item_t< K, T >( q, t, self, dense, alone, eps, pairs, cap, ps, dense_stack_limit, &it, &grid, &dense );
  // both objects' element slabs stored (dense contact): the walk that only reads them; else the one that computes the
  // slabs it tests from the vertices (unrolled when both objects have the same vertex count)
  if ( dense ) return walk_kernels< K, T, 0, true >::launch( it, grid, s );
  switch ( q.V == t.V ? q.V : 0 )
  {
    case 3: return walk_kernels< K, T, 3, false >::launch( it, grid, s );
    case 4: return walk_kernels< K, T, 4, false >::launch( it, grid, s );
    case 8: return walk_kernels< K, T, 8, false >::launch( it, grid, s );
    default: return walk_kernels< K, T, 0, false >::launch( it, grid, s );
  }
}

template< int K, typename T >
cudaError_t launch_trav_batch_t(bool dense, uint32_t V, const batch_launch &b, cudaStream_t s)
{
  if ( dense ) return walk_kernels< K, T, 0, true >::launch_batch( b, s );
  switch ( V )
  {
    case 3: return walk_kernels< K, T, 3, false >::launch_batch( b, s );
    case 4: return walk_kernels< K, T, 4, false >::launch_batch( b, s );
    case 8: return walk_kernels< K, T, 8, false >::launch_batch( b, s );
    default: return walk_kernels< K, T, 0, false >::launch_batch( b, s );
  }
}

// The vertices of one element into registers: 16-byte loads when every element starts on a 16-byte boundary (an
// even vertex count, 48 bytes per vertex pair, and a 16-byte aligned array), else 8-byte loads. Half the load
// instructions of the recheck for tetrahedra and hexahedra (tet lattice: 1.88 -> 1.65 ms at 18-DOP).
template< int V >
__device__ __forceinline__ void load_verts(const double *p, bool vec16, double *x)
{
  if constexpr ( V % 2 == 0 )
  {
    if ( vec16 )
    {
#pragma unroll
      for ( int k = 0; k < V * 3; k += 2 )
      {
        const double2 t = __ldg( reinterpret_cast< const double2 * >( p + k ) );
        x[k] = t.x;
        x[k + 1] = t.y;
      }
      return;
    }
  }
#pragma unroll
  for ( int k = 0; k < V * 3; ++k ) x[k] = __ldg( p + k );
}

constexpr int kRecheckThreads = 256;
constexpr int kRecheckBuf = 128;  // buffered pairs per warp: drained once more than 96 are held

// The candidate count is read on the device: no host round trip between traversal and recheck.
__device__ __forceinline__ uint64_t candidates(const recheck_args &args)
{
  return min( static_cast< uint64_t >( *reinterpret_cast< volatile unsigned long long * >( &args.ps->count ) ), args.cand_cap );
}

// K7: FP64 overlap of both elements from their vertices. With both vertex counts known at compile time, the
// comparison-only projections of overlap64 (shared products, no products by 0 or 1, one epsilon shift per slab);
// otherwise slab64 slab by slab with early exit. Both give the outcome of comparing the FP64 slabs.
// One warp takes the groups of 32 candidates u0, u0 + step, ... below u1; wout: its pair buffer.
template< int K, int VA, int VB >
__device__ __forceinline__ void recheck_groups(const recheck_args &args, uint64_t u0, uint64_t u1, uint64_t step, uint2 *wout)
{
  const double *__restrict__ va = args.va;
  const uint32_t Var = args.Va;
  const double *__restrict__ vb = args.vb;
  const uint32_t Vbr = args.Vb;
  const double eps = args.eps;
  const uint2 *__restrict__ cand = args.cand;
  uint2 *out = args.out;
  const uint64_t cap = args.cap;
  pair_scalars *ps = args.ps;
  constexpr int D = K / 2;
  const uint64_t ncand = candidates( args );
  const int Va = VA > 0 ? VA : static_cast< int >( Var );
  const int Vb = VB > 0 ? VB : static_cast< int >( Vbr );
  const bool vec16 = ( ( reinterpret_cast< uintptr_t >( va ) | reinterpret_cast< uintptr_t >( vb ) ) & 15 ) == 0;
  // Confirmed pairs collect in a per-warp buffer in shared memory and leave through one atomic reservation per
  // 97-128 pairs, with coalesced stores (one same-address atomic per 32 candidates made the kernel wait on the
  // counter's round trip).
  const unsigned lane = threadIdx.x & 31u, lt = ( 1u << lane ) - 1u;
  uint32_t nout = 0;
  auto drain = [&]() {
    __syncwarp();
    unsigned long long base = 0;
    if ( lane == 0 && nout ) base = atomicAdd( &ps->count2, static_cast< unsigned long long >( nout ) );
    base = __shfl_sync( 0xffffffffu, base, 0 );
    for ( uint32_t j = lane; j < nout; j += 32 )
      if ( base + j < cap ) out[base + j] = wout[j];
    __syncwarp();
    nout = 0;
  };
  for ( uint64_t u = u0; u < u1; u += step )
  {
    const uint64_t p = 32 * u + lane;
    const bool valid = p < ncand;
    const uint2 c = valid ? __ldg( cand + p ) : make_uint2( 0u, 0u );
    bool ok = valid;
    const double *pa = va + static_cast< size_t >( c.x ) * Va * 3;
    const double *pb = vb + static_cast< size_t >( c.y ) * Vb * 3;
    double xa[VA > 0 ? VA * 3 : 24], xb[VB > 0 ? VB * 3 : 24];
    if constexpr ( VA > 0 && VB > 0 )
    {
      if ( valid )
      {
        load_verts< VA >( pa, vec16, xa );
        load_verts< VB >( pb, vec16, xb );
        ok = overlap64< K, VA, VB >( xa, xb, eps );
      }
    } else {
      (void)xa;
      (void)xb;
#pragma unroll
      for ( int a = 0; a < D; ++a )
      {
        if ( !ok ) break;
        double alo = 0, ahi = 0, blo = 0, bhi = 0;
        for ( int v = 0; v < Va; ++v )
        {
          const double q[3] = { __ldg( pa + 3 * v ), __ldg( pa + 3 * v + 1 ), __ldg( pa + 3 * v + 2 ) };
          double l, h;
          slab64< K >( q, 1, a, eps, l, h );
          alo = v ? std_min( alo, l ) : l;
          ahi = v ? std_max( ahi, h ) : h;
        }
        for ( int v = 0; v < Vb; ++v )
        {
          const double q[3] = { __ldg( pb + 3 * v ), __ldg( pb + 3 * v + 1 ), __ldg( pb + 3 * v + 2 ) };
          double l, h;
          slab64< K >( q, 1, a, eps, l, h );
          blo = v ? std_min( blo, l ) : l;
          bhi = v ? std_max( bhi, h ) : h;
        }
        ok = alo < bhi && blo < ahi;
      }
    }
    const unsigned bal = __ballot_sync( 0xffffffffu, ok );
    if ( ok ) wout[nout + static_cast< unsigned >( __popc( bal & lt ) )] = c;
    nout += static_cast< uint32_t >( __popc( bal ) );
    if ( nout > kRecheckBuf - 32 ) drain();
  }
  drain();
}

template< int K, int VA, int VB >
__device__ void recheck_body(const recheck_args &args, uint32_t bid, uint32_t nblk)
{
  __shared__ uint2 s_out[kRecheckThreads / 32][kRecheckBuf];
  constexpr uint32_t W = kRecheckThreads / 32;
  recheck_groups< K, VA, VB >( args, static_cast< uint64_t >( bid ) * W + ( threadIdx.x >> 5 ), ( candidates( args ) + 31 ) / 32,
                               static_cast< uint64_t >( nblk ) * W, s_out[threadIdx.x >> 5] );
}

// ---- the scenes of a batch in one launch ----------------------------------------------------------------------
//
// Each scene's pair count is known on the device only, and most scenes of a batch have few or none: a launch with
// blocks for every scene's capacity spends its time on starting blocks that find nothing (496 pairs of 32 bodies, most
// of them apart: 294,000 blocks, 1.0 ms for the recheck and 0.24 ms for the ids over the groups of a batch). A grid of
// the resident blocks instead forms the running sum of the scenes' counts, kSceneTile scenes at a time, and divides the
// sum.
constexpr int kSceneTile = 2 * kRecheckThreads;

// pre[0 .. count] = the exclusive running sum of f(0 .. count - 1), by a block of kRecheckThreads threads.
template< typename F >
__device__ __forceinline__ void scene_sum(int count, F f, unsigned long long *pre)
{
  __shared__ unsigned long long s_warp[kRecheckThreads / 32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const unsigned long long v0 = 2 * t < count ? f( 2 * t ) : 0ull, v1 = 2 * t + 1 < count ? f( 2 * t + 1 ) : 0ull;
  unsigned long long inc = v0 + v1;
#pragma unroll
  for ( int o = 1; o < 32; o <<= 1 )
  {
    const unsigned long long y = __shfl_up_sync( 0xffffffffu, inc, o );
    if ( lane >= o ) inc += y;
  }
  if ( lane == 31 ) s_warp[w] = inc;
  __syncthreads();
  for ( int k = 0; k < w; ++k ) inc += s_warp[k];
  if ( t == 0 ) pre[0] = 0ull;
  if ( 2 * t < count ) pre[2 * t + 1] = inc - v1;
  if ( 2 * t + 1 < count ) pre[2 * t + 2] = inc;
  __syncthreads();
}

// The last scene whose sum is <= u (u below the total).
__device__ __forceinline__ int scene_of(const unsigned long long *pre, int count, unsigned long long u)
{
  int lo = 0, hi = count - 1;
  while ( lo < hi )
  {
    const int mid = ( lo + hi + 1 ) >> 1;
    if ( pre[mid] <= u ) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// The grid: the resident blocks (2 per SM), or the blocks that the scenes' capacities can occupy if those are fewer. The
// groups of a batch run beside one another, and a grid of small scenes that took every SM's registers held the others up
// (16 scenes of 4,000 triangles with the FP32 filter 304 -> 271 us a call, 300 of 200 1,268 -> 1,233).
uint32_t scene_grid(const batch_launch &b)
{
  const uint32_t most = static_cast< uint32_t >( device_sm_count() ) * 2;
  return b.blocks < most ? b.blocks : most;
}

// The recheck of n scenes: every warp takes an equal share of consecutive groups of 32 candidates.
template< int K, int VA, int VB >
__global__ void __launch_bounds__( kRecheckThreads, 2 ) k_recheck_scenes(const recheck_args *__restrict__ items, int n)
{
  constexpr uint32_t W = kRecheckThreads / 32;
  __shared__ uint2 s_out[W][kRecheckBuf];
  __shared__ unsigned long long s_pre[kSceneTile + 1];
  const unsigned long long warps = static_cast< unsigned long long >( gridDim.x ) * W, w = blockIdx.x * W + ( threadIdx.x >> 5 );
  for ( int t0 = 0; t0 < n; t0 += kSceneTile )
  {
    const int count = min( kSceneTile, n - t0 );
    scene_sum( count, [&](int s) -> unsigned long long { return ( candidates( items[t0 + s] ) + 31 ) / 32; }, s_pre );
    const unsigned long long total = s_pre[count], end = total * ( w + 1 ) / warps;
    for ( unsigned long long u = total * w / warps; u < end; )
    {
      const int s = scene_of( s_pre, count, u );
      const unsigned long long last = min( end, s_pre[s + 1] );
      const recheck_args a = items[t0 + s];
      recheck_groups< K, VA, VB >( a, u - s_pre[s], last - s_pre[s], 1, s_out[threadIdx.x >> 5] );
      u = last;
    }
    __syncthreads();  // the next tile reuses the sums
  }
}

// grid-stride over the candidates (their count is read on the device): at most 4 blocks per SM
uint32_t recheck_grid(uint64_t ncand)
{
  const uint64_t blocks = ( ncand + kRecheckThreads - 1 ) / kRecheckThreads;
  const uint64_t capb = static_cast< uint64_t >( device_sm_count() ) * 4;
  return static_cast< uint32_t >( blocks < capb ? ( blocks ? blocks : 1 ) : capb );
}

template< int K >
cudaError_t recheck_k(const recheck_args &a, cudaStream_t s)
{
  const uint32_t grid = recheck_grid( a.cand_cap );
  if ( a.Va == 3 && a.Vb == 3 ) k_single< recheck_args, recheck_body< K, 3, 3 >, kRecheckThreads, 2 ><<< grid, kRecheckThreads, 0, s >>>( a );
  else if ( a.Va == 4 && a.Vb == 4 ) k_single< recheck_args, recheck_body< K, 4, 4 >, kRecheckThreads, 2 ><<< grid, kRecheckThreads, 0, s >>>( a );
  else if ( a.Va == 8 && a.Vb == 8 ) k_single< recheck_args, recheck_body< K, 8, 8 >, kRecheckThreads, 2 ><<< grid, kRecheckThreads, 0, s >>>( a );
  else k_single< recheck_args, recheck_body< K, 0, 0 >, kRecheckThreads, 2 ><<< grid, kRecheckThreads, 0, s >>>( a );
  return cudaGetLastError();
}

template< int K >
cudaError_t recheck_batch_k(uint32_t V, const batch_launch &b, cudaStream_t s)
{
  const recheck_args *it = static_cast< const recheck_args * >( b.items );
  const uint32_t grid = scene_grid( b );
  if ( V == 3 ) k_recheck_scenes< K, 3, 3 ><<< grid, kRecheckThreads, 0, s >>>( it, b.nitems );
  else if ( V == 4 ) k_recheck_scenes< K, 4, 4 ><<< grid, kRecheckThreads, 0, s >>>( it, b.nitems );
  else if ( V == 8 ) k_recheck_scenes< K, 8, 8 ><<< grid, kRecheckThreads, 0, s >>>( it, b.nitems );
  else k_recheck_scenes< K, 0, 0 ><<< grid, kRecheckThreads, 0, s >>>( it, b.nitems );
  return cudaGetLastError();
}

__global__ void k_gid_pairs(const uint2 *__restrict__ pairs, uint64_t count, const uint64_t *__restrict__ gid_a,
                            const uint64_t *__restrict__ gid_b, int normalize, uint64_t *__restrict__ out)
{
  for ( uint64_t p = static_cast< uint64_t >( blockIdx.x ) * blockDim.x + threadIdx.x; p < count;
        p += static_cast< uint64_t >( gridDim.x ) * blockDim.x )
  {
    uint2 c = pairs[p];
    if ( normalize && c.x > c.y ) c = make_uint2( c.y, c.x );
    const uint64_t a = gid_a ? __ldg( gid_a + c.x ) : c.x;
    const uint64_t b = gid_b ? __ldg( gid_b + c.y ) : c.y;
    reinterpret_cast< ulonglong2 * >( out )[p] = make_ulonglong2( a, b );
  }
}

// k_gid_pairs with the count read on the device (at most cap): for launches whose count is unknown when they are
// enqueued (batched scenes in a CUDA graph).
__device__ __forceinline__ uint64_t gid_count(const gid_args &a)
{
  return min( static_cast< uint64_t >( *reinterpret_cast< const volatile unsigned long long * >( a.count ) ), a.cap );
}

__device__ __forceinline__ void write_ids(const gid_args &a, uint64_t p)
{
  uint2 c = a.pairs[p];
  if ( a.normalize && c.x > c.y ) c = make_uint2( c.y, c.x );
  const uint64_t ga = a.gid_a ? __ldg( a.gid_a + c.x ) : c.x;
  const uint64_t gb = a.gid_b ? __ldg( a.gid_b + c.y ) : c.y;
  reinterpret_cast< ulonglong2 * >( a.out )[p] = make_ulonglong2( ga, gb );
}

__device__ void gid_dev_body(const gid_args &a, uint32_t bid, uint32_t nblk)
{
  const uint64_t n = gid_count( a );
  for ( uint64_t p = static_cast< uint64_t >( bid ) * blockDim.x + threadIdx.x; p < n;
        p += static_cast< uint64_t >( nblk ) * blockDim.x )
    write_ids( a, p );
}

// The same for n scenes in one launch (see "the scenes of a batch in one launch").
__global__ void __launch_bounds__( kRecheckThreads ) k_gid_scenes(const gid_args *__restrict__ items, int n)
{
  __shared__ unsigned long long s_pre[kSceneTile + 1];
  for ( int t0 = 0; t0 < n; t0 += kSceneTile )
  {
    const int count = min( kSceneTile, n - t0 );
    scene_sum( count, [&](int s) -> unsigned long long { return gid_count( items[t0 + s] ); }, s_pre );
    const unsigned long long total = s_pre[count];
    for ( unsigned long long u = static_cast< unsigned long long >( blockIdx.x ) * kRecheckThreads + threadIdx.x; u < total;
          u += static_cast< unsigned long long >( gridDim.x ) * kRecheckThreads )
    {
      const int s = scene_of( s_pre, count, u );
      write_ids( items[t0 + s], u - s_pre[s] );
    }
    __syncthreads();  // the next tile reuses the sums
  }
}

// dst[i] = *src[i]: the error words of many objects in one copy.
__global__ void k_gather_words(const int *const *__restrict__ src, int n, int *__restrict__ dst)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if ( i < n ) dst[i] = *reinterpret_cast< const volatile int * >( src[i] );
}

}  // namespace

uint32_t scene_blocks(uint64_t cap)
{
  const uint64_t blocks = ( cap + kRecheckThreads - 1 ) / kRecheckThreads;
  return static_cast< uint32_t >( blocks < 1 ? 1 : ( blocks < 148 * 2 ? blocks : 148 * 2 ) );
}

static uint32_t gid_pairs_dev_blocks(uint64_t cap)
{
  const uint64_t blocks = ( cap + 255 ) / 256;
  return static_cast< uint32_t >( blocks < 148 * 2 ? ( blocks ? blocks : 1 ) : 148 * 2 );
}

cudaError_t launch_gid_pairs_dev(const uint2 *pairs, const unsigned long long *count, uint64_t cap,
                                 const uint64_t *gid_a, const uint64_t *gid_b, bool normalize, uint64_t *out,
                                 cudaStream_t s)
{
  if ( cap == 0 ) return cudaSuccess;
  const gid_args a{ pairs, count, cap, gid_a, gid_b, normalize ? 1 : 0, out };
  k_single< gid_args, gid_dev_body, 256, 1 ><<< gid_pairs_dev_blocks( cap ), 256, 0, s >>>( a );
  return cudaGetLastError();
}

cudaError_t launch_gid_pairs_dev_batch(const batch_launch &b, cudaStream_t s)
{
  if ( !b.nitems ) return cudaSuccess;
  k_gid_scenes<<< scene_grid( b ), kRecheckThreads, 0, s >>>( static_cast< const gid_args * >( b.items ), b.nitems );
  return cudaGetLastError();
}

cudaError_t launch_gather_words(const int *const *src, int n, int *dst, cudaStream_t s)
{
  if ( n == 0 ) return cudaSuccess;
  k_gather_words<<< ( n + 255 ) / 256, 256, 0, s >>>( src, n, dst );
  return cudaGetLastError();
}

cudaError_t launch_traverse(int K, bool fp32, tree_view q, tree_view t, bool self, bool dense, double eps, uint2 *pairs,
                            uint64_t cap, pair_scalars *ps, cudaStream_t s, int dense_stack_limit, bool alone)
{
  switch ( K )
  {
    case 6: return fp32 ? launch_trav_t< 6, float >( q, t, self, dense, eps, pairs, cap, ps, s, dense_stack_limit, alone )
                        : launch_trav_t< 6, double >( q, t, self, dense, eps, pairs, cap, ps, s, dense_stack_limit, alone );
    case 18: return fp32 ? launch_trav_t< 18, float >( q, t, self, dense, eps, pairs, cap, ps, s, dense_stack_limit, alone )
                         : launch_trav_t< 18, double >( q, t, self, dense, eps, pairs, cap, ps, s, dense_stack_limit, alone );
    case 26: return fp32 ? launch_trav_t< 26, float >( q, t, self, dense, eps, pairs, cap, ps, s, dense_stack_limit, alone )
                         : launch_trav_t< 26, double >( q, t, self, dense, eps, pairs, cap, ps, s, dense_stack_limit, alone );
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_recheck(int K, const double *verts_a, uint32_t Va, const double *verts_b, uint32_t Vb, double eps,
                           const uint2 *cand, uint64_t ncand, uint2 *out, uint64_t cap, pair_scalars *ps,
                           cudaStream_t s)
{
  const recheck_args a{ verts_a, Va, verts_b, Vb, eps, cand, ncand, out, cap, ps };
  switch ( K )
  {
    case 6: return recheck_k< 6 >( a, s );
    case 18: return recheck_k< 18 >( a, s );
    case 26: return recheck_k< 26 >( a, s );
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_recheck_batch(int K, uint32_t V, const batch_launch &b, cudaStream_t s)
{
  if ( !b.nitems ) return cudaSuccess;
  switch ( K )
  {
    case 6: return recheck_batch_k< 6 >( V, b, s );
    case 18: return recheck_batch_k< 18 >( V, b, s );
    case 26: return recheck_batch_k< 26 >( V, b, s );
    default: return cudaErrorInvalidValue;
  }
}

void traverse_item(int K, bool fp32, tree_view q, tree_view t, bool self, bool dense, double eps, uint2 *pairs,
                   uint64_t cap, pair_scalars *ps, int dense_stack_limit, trav_item *item, uint32_t *blocks,
                   bool *dense_out)
{
  // the item's fields do not depend on K or the slab type; only the grid depends on K through nothing either
  if ( fp32 ) trav_item_t< 18, float >( q, t, self, dense, false, eps, pairs, cap, ps, dense_stack_limit, item, blocks, dense_out );
  else trav_item_t< 18, double >( q, t, self, dense, false, eps, pairs, cap, ps, dense_stack_limit, item, blocks, dense_out );
  (void)K;
}

cudaError_t launch_traverse_batch(int K, bool fp32, bool dense, uint32_t V, const batch_launch &b, cudaStream_t s)
{
  if ( !b.nitems ) return cudaSuccess;
  switch ( K )
  {
    case 6: return fp32 ? launch_trav_batch_t< 6, float >( dense, V, b, s ) : launch_trav_batch_t< 6, double >( dense, V, b, s );
    case 18: return fp32 ? launch_trav_batch_t< 18, float >( dense, V, b, s ) : launch_trav_batch_t< 18, double >( dense, V, b, s );
    case 26: return fp32 ? launch_trav_batch_t< 26, float >( dense, V, b, s ) : launch_trav_batch_t< 26, double >( dense, V, b, s );
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_gid_pairs(const uint2 *pairs, uint64_t count, const uint64_t *gid_a, const uint64_t *gid_b,
                             bool normalize, uint64_t *out, cudaStream_t s)
{
  if ( count == 0 ) return cudaSuccess;
  const uint64_t blocks = ( count + 255 ) / 256;
  const unsigned grid = static_cast< unsigned >( blocks < 148 * 8 ? blocks : 148 * 8 );
  k_gid_pairs<<< grid, 256, 0, s >>>( pairs, count, gid_a, gid_b, normalize ? 1 : 0, out );
  return cudaGetLastError();
}

}  // namespace bvhg
