// Waits of a launch's blocks for one another, for the units whose blocks trade cells. Every such
// wait is bounded. A block whose wait runs out has no usable iterate from there on: what it stores,
// hands to other blocks or adds to a sum is NaN, so that no finite value depends on it, and the
// unit counts the block (sg_lost_waits), which a call that returns before its kernels have run
// cannot report.
//
// In the bounds-check build a test can name a block that gives up each wait at once
// (sg_bounds_lose_waits); in the normal build lose_waits is `false` and compiles away.
#pragma once

#include "common.cuh"

namespace sg {

static __device__ unsigned int g_lost_waits;  // one word per translation unit

// At the block's end, by every thread: s_lost is the block's mark, settled by a barrier. (Counted
// in the poll loops, the atomics cost the Gauss-Seidel chain 2 %.)
__device__ __forceinline__ void count_lost_wait(int s_lost) {
  if (s_lost && threadIdx.x == 0) atomicAdd(&g_lost_waits, 1u);
}

#if SG_BOUNDS_CHECK
static __device__ int g_lose_block = -1;
__device__ __forceinline__ bool lose_waits(int block) { return block == *(volatile int*)&g_lose_block; }
#define SG_SET_LOSE_BLOCK(block) \
  (cudaMemcpyToSymbol(::sg::g_lose_block, &block, sizeof(int)) == cudaSuccess ? SG_OK : SG_ERR_CUDA)
#else
__device__ __forceinline__ bool lose_waits(int) { return false; }
#define SG_SET_LOSE_BLOCK(block) ((void)block, SG_ERR_ARG)
#endif

}  // namespace sg

#define SG_WAITS_ACCESSOR(unit)                                                                   \
  extern "C" int sg_lost_waits_##unit(unsigned* count, int clear) {                               \
    if (cudaMemcpyFromSymbol(count, ::sg::g_lost_waits, sizeof(unsigned)) != cudaSuccess)         \
      return SG_ERR_CUDA;                                                                         \
    const unsigned zero = 0;                                                                      \
    if (clear && cudaMemcpyToSymbol(::sg::g_lost_waits, &zero, sizeof(unsigned)) != cudaSuccess)  \
      return SG_ERR_CUDA;                                                                         \
    return SG_OK;                                                                                 \
  }                                                                                               \
  extern "C" int sg_lose_waits_##unit(int block) { return SG_SET_LOSE_BLOCK(block); }
