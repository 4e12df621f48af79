// batch.cuh — the launches of one kernel for many objects (or scenes) as a single launch.
//
// Each kernel of the pipeline is written as a __device__ body over an argument struct, its block index and its block
// count. The per-object launch runs the body with blockIdx.x and gridDim.x; a batched launch runs the blocks of many
// items back to back: item i owns blocks [starts[i], starts[i + 1]) of the grid, each with the block count the
// per-object launch would have used. A block finds its item by binary search over `starts` and runs the item's body,
// so every item computes exactly what its own launch would have computed; only the number of launches changes.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace bvhg {

// The item owning grid block b: the last i with starts[i] <= b (starts ascending, starts[0] = 0).
__device__ __forceinline__ int batch_item_of(const uint32_t *__restrict__ starts, int n, uint32_t b)
{
  int lo = 0, hi = n - 1;
  while ( lo < hi )
  {
    const int mid = ( lo + hi + 1 ) >> 1;
    if ( __ldg( starts + mid ) <= b ) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// One launch over the blocks of all items: items[i] are item i's arguments.
template< typename Args, void ( *Body )( const Args &, uint32_t, uint32_t ), int THREADS, int MIN_BLOCKS >
__global__ void __launch_bounds__( THREADS, MIN_BLOCKS ) k_batched(const Args *__restrict__ items,
                                                                   const uint32_t *__restrict__ starts, int nitems)
{
  __shared__ int s_item;
  if ( threadIdx.x == 0 ) s_item = batch_item_of( starts, nitems, blockIdx.x );
  __syncthreads();
  const int i = s_item;
  const uint32_t b0 = __ldg( starts + i );
  const Args a = items[i];
  Body( a, blockIdx.x - b0, __ldg( starts + i + 1 ) - b0 );
}

// One per-object launch of a body. An object's kernels follow one another in a stream, each reading what the last one
// wrote. For a small object launch_chained() lets the next kernel's blocks start while this one's still run, and every
// kernel waits here until the kernels before it have completed and their writes are visible (so a chain of waiting
// kernels is ordered as a plain one). What overlaps is the launch itself: the 12 kernels of a build of 10,000 triangles
// take a few microseconds each, and a step of two such objects went from 412 to 381 us, one of 200,003 tetrahedra from
// 467 to 458 us, two blocks of 512 hexahedra from 356 to 345 us. Above kChainElements the launches are plain: there the
// waiting blocks take the place of the other object's kernels (1.3M and 1.0M triangles 526 -> 554 us with the chain, a
// refit of 9.4M triangles 682 -> 713 us).
constexpr uint64_t kChainElements = 1u << 19;
constexpr uint32_t kChainBlocks = 296;  // 2 blocks for each of 148 SMs: beyond it the successor's blocks start as these leave

template< typename Args, void ( *Body )( const Args &, uint32_t, uint32_t ), int THREADS, int MIN_BLOCKS >
__global__ void __launch_bounds__( THREADS, MIN_BLOCKS ) k_single(const Args a)
{
  if ( gridDim.x <= kChainBlocks ) asm volatile( "griddepcontrol.launch_dependents;" ::: "memory" );
  asm volatile( "griddepcontrol.wait;" ::: "memory" );
  Body( a, blockIdx.x, gridDim.x );
}

// Launches a per-object kernel whose predecessor in the stream is the previous kernel of the object (n elements).
template< typename Args >
cudaError_t launch_chained(uint64_t n, void ( *kernel )( Args ), uint32_t grid, uint32_t threads, size_t smem, cudaStream_t s,
                           const Args &a)
{
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3( grid );
  cfg.blockDim = dim3( threads );
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = n <= kChainElements ? 1 : 0;
  return cudaLaunchKernelEx( &cfg, kernel, a );
}

// Host side: a batched launch description (item arguments and block starts on the device, built when a batch graph
// is captured).
struct batch_launch
{
  const void *items = nullptr;     // device array of the kernel's argument structs
  const uint32_t *starts = nullptr;  // device array of nitems + 1 block starts
  int nitems = 0;
  uint32_t blocks = 0;             // starts[nitems]
};

}  // namespace bvhg
