/* spp_grid.cuh -- barrier and scan of a cooperative launch (the resident
 * runs, kernels_run.cu and kernels_vrun.cu). */
#ifndef SPP_GRID_CUH
#define SPP_GRID_CUH
#include "spp_internal.cuh"
#include "spp_list.cuh"

namespace {

/* polls of a barrier's counter before a block gives up (a poll takes about
 * 0.7 us: seconds; a barrier is normally met within microseconds) */
#ifndef SPP_RUN_WAIT_LIMIT
#define SPP_RUN_WAIT_LIMIT (1 << 22)
#endif
constexpr int RUN_WAIT_LIMIT = SPP_RUN_WAIT_LIMIT;   /* 0: every wait gives up at once (a test's build) */
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ unsigned ld_relaxed(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

/* One arrival of the block at the grid barrier: every write of the block
 * before it is visible to a block that has waited for it.  Thread 0 calls,
 * after a __syncthreads. */
__device__ __forceinline__ void grid_arrive(Ctl* ctl) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&ctl->run_bar) : "memory");
}

/* Thread 0: waits until the counter has reached target, or gives up. */
__device__ __forceinline__ bool grid_wait(Ctl* ctl, unsigned target) {
  for (int it = 0; it < RUN_WAIT_LIMIT; ++it)
    if (ld_acquire(&ctl->run_bar) >= target) return true;
  atomicOr(&ctl->run_timeout, 1u);
  return false;
}

/* Exclusive scan of n counts (n a multiple of 4, both arrays 16-byte
 * aligned) by the whole grid: each block sums, then scans, its own range.
 * The counts are complete (a barrier lies behind); the starts are visible
 * after the caller's next barrier.  sums: one word per block. */
template <class Barrier>
__device__ __forceinline__ bool grid_scan(const uint32_t* count, uint32_t* start, uint32_t n, uint32_t* sums,
                                          Barrier barrier) {
  const int T = blockDim.x, tid = threadIdx.x;
  const uint32_t per_block = ((n + gridDim.x - 1) / gridDim.x + 3u) & ~3u;
  const uint32_t c0 = min(per_block * blockIdx.x, n), c1 = min(c0 + per_block, n);
  uint32_t sum = 0u;
  for (uint32_t c = c0 + 4u * tid; c < c1; c += 4u * T) {
    const uint4 v = *reinterpret_cast<const uint4*>(count + c);
    sum += (v.x + v.y) + (v.z + v.w);
  }
  uint32_t total;
  block_exclusive_scan(sum, &total);
  if (tid == 0) sums[blockIdx.x] = total;
  if (!barrier()) return false;
  uint32_t before = 0u;
  for (uint32_t b = tid; b < blockIdx.x; b += T) before += sums[b];
  uint32_t carry;
  block_exclusive_scan(before, &carry);
  for (uint32_t cb = c0; cb < c1; cb += 4u * T) {
    __syncthreads();
    const uint32_t c = cb + 4u * tid;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (c < c1) v = *reinterpret_cast<const uint4*>(count + c);
    const uint32_t e = carry + block_exclusive_scan((v.x + v.y) + (v.z + v.w), &total);
    if (c < c1)
      *reinterpret_cast<uint4*>(start + c) = make_uint4(e, e + v.x, e + v.x + v.y, e + v.x + v.y + v.z);
    carry += total;
  }
  return true;
}

}  // namespace
#endif
