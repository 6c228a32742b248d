/* spp_rebuild.cuh -- the neighbour-list rebuild inside a resident run
 * (kernels_run.cu, kernels_lrun.cu). */
#ifndef SPP_REBUILD_CUH
#define SPP_REBUILD_CUH
#include "spp_grid.cuh"
#include "spp_list.cuh"

namespace {

/* Shared memory per thread: the list build's LIST_LOCAL slots, then the keys
 * of the long-list sort (RUN_SORT_MAX per warp); between rebuilds the same
 * bytes hold the first run_rows() entries of the thread's neighbour segment
 * (later entries are read from global memory): 32 of them, or 64 where the
 * list capacity (grown by flocks) says that segments run past 32 and one
 * block per SM leaves the room. */
constexpr int RUN_SORT_MAX = 512;
constexpr int RUN_SMEM = RUN_SORT_MAX * 8 / 32;
static_assert(RUN_SMEM >= LIST_LOCAL * 4, "the build's slots");
constexpr int RUN_ROWS = RUN_SMEM / 4, RUN_ROWS_LONG = 64;
__host__ __device__ inline int run_rows(int cap, int lanes, int per_sm) {
  return per_sm == 1 && cap > 3 * lanes * RUN_ROWS / 4 ? RUN_ROWS_LONG : RUN_ROWS;
}
/* Segments from this length on (the longest of a warp) are walked with more
 * neighbours in flight. */
constexpr int RUN_LONG = 12;

/* A queued list (longer than LIST_LOCAL) put in order by the calling warp, as
 * sort_queued_list (spp_list.cuh) does, by a bitonic network over keys in
 * the warp's shared memory: loops instead of registers, a tenth of the code. */
__device__ __forceinline__ void run_sort_list(const SppConsts& k, const DevState& d, int i, unsigned long long* keys) {
  const int lane = threadIdx.x & 31;
  const int m = d.nn[i];
  if (m > RUN_SORT_MAX) {
    sort_list_in_place(k, d, i, m);
    return;
  }
  int size = 32;
  while (size < m) size <<= 1;
  for (int q = lane; q < size; q += 32) {
    unsigned long long key = ~0ull;
    if (q < m) {
      int32_t j = d.nbr[(size_t)q * d.n + i];
      if (!spp_index_ok(d.ctl, j, d.n)) j = i;
      key = ((unsigned long long)spp_list_order(&k, d.id_alt[j]) << 32) | (unsigned long long)(uint32_t)j;
    }
    keys[q] = key;
  }
  __syncwarp();
  for (int run = 2; run <= size; run <<= 1)
    for (int stride = run >> 1; stride > 0; stride >>= 1) {
      for (int e = lane; e < size / 2; e += 32) {
        const int lo = 2 * e - (e & (stride - 1)), hi = lo + stride;
        const unsigned long long a = keys[lo], b = keys[hi];
        if (((lo & run) == 0) == (a > b)) {
          keys[lo] = b;
          keys[hi] = a;
        }
      }
      __syncwarp();
    }
  for (int q = lane; q < m; q += 32) d.nbr[(size_t)q * d.n + i] = (int32_t)(uint32_t)keys[q];
  __syncwarp();
}

enum { RUN_LOST = 0, RUN_BUILT = 1, RUN_FROZEN = 2 };

/* The rebuild inside a resident run, the phases of enqueue_rebuild (api.cu)
 * with a grid barrier between them: the owners' registers (position p,
 * heading th0, id pid) are scattered into cell order, and the lists are
 * built from that copy.  cell_count is all zero on entry and on return.
 * One copy per lane count, called: it runs every ten steps or so, and
 * inlined it would cost the step loop registers. */
template <int LANES>
__device__ __noinline__ int run_rebuild(const SppConsts& k, const DevState& d, int i, bool head, float4 p,
                                        float th0, uint32_t pid, unsigned long long* keycol, unsigned* target,
                                        unsigned* s_word) {
  const int T = blockDim.x, tid = threadIdx.x, n = d.n;
  const int gthreads = gridDim.x * T, gtid = blockIdx.x * T + tid;
  Ctl* const ctl = d.ctl;
  /* arrive and wait in one; false when the block must leave */
  auto barrier = [&]() -> bool {
    *target += gridDim.x;
    __syncthreads();
    if (tid == 0) {
      grid_arrive(ctl);
      *s_word = grid_wait(ctl, *target);
    }
    __syncthreads();
    return *s_word != 0u;
  };
  uint32_t key = 0u, rank = 0u;
  if (gtid == 0) ctl->long_n = 0u;
  if (head) {
    int cx, cy;
    key = cell_key(k, d, p.x, p.y, &cx, &cy);
    if (!spp_index_ok(ctl, key, d.n_keys)) key = 0u;
    rank = atomicAdd(&d.cell_count[key], 1u);
  }
  if (!barrier()) return RUN_LOST;
  if (!grid_scan(d.cell_count, d.cell_start, d.n_keys, d.run_sums, barrier)) return RUN_LOST;
  if (!barrier()) return RUN_LOST;
  if (head) {
    const uint32_t dst = d.cell_start[key] + rank;
    if (spp_index_ok(ctl, dst, n)) {
      d.pos_alt[dst] = p;
      d.theta_alt[dst] = th0;
      d.img_alt[dst] = d.img[i];
      d.id_alt[dst] = pid;
    }
  }
  if (!barrier()) return RUN_LOST;
  {
    /* one thread per particle: the block's particles, packed */
    const int ib = blockIdx.x * (T / LANES) + tid;
    uint32_t cnt = 0u;
    if (tid < T / LANES && ib < n) {
      const float4 q = d.pos_alt[ib];
      cnt = build_particle_list<LANES>(k, d, ib, q, reinterpret_cast<uint32_t*>(keycol - tid) + tid, T);
      adopt_sorted_particle(d, ib, q);
    }
    note_list_lengths(d, cnt);
    if (gtid == 0) atomicAdd(&ctl->n_rebuilds, 1u);
  }
  if (!barrier()) return RUN_LOST;
  const uint32_t longs = *reinterpret_cast<volatile uint32_t*>(&ctl->long_n);
  const uint32_t frozen = *reinterpret_cast<volatile uint32_t*>(&ctl->frozen);
  if (longs > 0u) {
    for (uint32_t w = (uint32_t)(gtid >> 5); w < longs; w += (uint32_t)(gthreads >> 5)) {
      const int who = d.long_q[w];
      if (spp_index_ok(ctl, who, n)) run_sort_list(k, d, who, keycol - tid + (tid >> 5) * RUN_SORT_MAX);
    }
    if (!barrier()) return RUN_LOST;
  }
  /* the counts of the next rebuild (at least one barrier away) */
  for (uint32_t c = gtid; c < d.n_keys; c += gthreads) d.cell_count[c] = 0u;
  return frozen ? RUN_FROZEN : RUN_BUILT;
}

}  // namespace
#endif
