/*
 * kernels_cells.cu -- cell binning and neighbour lists on sm_103a.
 *
 * Replaces Box::Update_Cells (serial/box.h:107-134, parallel/node.h:710-911)
 * and Box::Update_Neighbor_List (serial/box.h:137-179, shared/cell.h:74-103).
 * The reference pushes particle ids into a vector<int> per cell and keeps a
 * half Verlet list per particle, rebuilt every cell_update_period steps.
 * Here:
 *   1. bin_count: one thread per particle computes its cell's Morton key and
 *      takes a slot in that cell with an atomicAdd.
 *   2. scan: exclusive prefix sum of the per-key counts (two passes).
 *   3. scatter: every particle's state moves to its cell-ordered slot, so
 *      that spatial neighbours are neighbours in memory (Morton order keeps
 *      2-D tiles of cells contiguous).
 *   4. build_list: one thread per particle scans the 3x3 cells around it and
 *      records every particle within r_list = r_cut + skin (full list: each
 *      pair appears in both particles' lists, so the force kernels gather
 *      without atomics), column-major nbr[slot * n + i], each list sorted by
 *      particle id so that the force kernels sum in a reproducible order.
 * Order inside a cell depends on atomic arrival order and is therefore not
 * deterministic; the sorted lists (Verlet models) and the order-independent
 * fixed-point sums (Vicsek models) keep the physics deterministic.
 */
#include "spp_internal.cuh"
#include "spp_list.cuh"
#include "spp_pack.cuh"

namespace {

/* One atomic per particle: cells hold one or two, so grouping a warp's equal
 * keys first (__match_any_sync) saved few atomics and took 16.4 us at N =
 * 1,048,576 against 8.5. */
__global__ void __launch_bounds__(SPP_BLOCK) k_bin_count(SppConsts k, DevState d) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) d.ctl->long_n = 0u;   /* the long-list queue of this rebuild (k_build_list) */
  if (i >= d.n) return;
  float4 p = d.pos[i];
  int cx, cy;
  uint32_t key = cell_key(k, d, p.x, p.y, &cx, &cy);
  if (!spp_index_ok(d.ctl, key, d.n_keys)) key = 0u;
  d.key[i] = key;
  d.rank[i] = atomicAdd(&d.cell_count[key], 1u);
}

/* ---- exclusive scan of cell_count into cell_start ---------------------- */
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_PER_THREAD = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_PER_THREAD;

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const uint32_t* __restrict__ in,
                                                              uint32_t n, uint32_t* block_sums) {
  uint32_t base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER_THREAD;
  uint32_t s = 0;
#pragma unroll
  for (int q = 0; q < SCAN_PER_THREAD; ++q)
    if (base + q < n) s += in[base + q];
  s = __reduce_add_sync(0xffffffffu, s);
  __shared__ uint32_t ws[SCAN_THREADS / 32];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    uint32_t t = ws[threadIdx.x];
    t = __reduce_add_sync(0xffffffffu, t);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = t;
  }
}

/* The second pass: a block takes its offset from the sums of the blocks before
 * it (a million cells have 256; a launch that scans the sums first costs
 * more).  NEXT also adds the total as entry n and clears the counts for the
 * next step of a batch.  counts and out start on 16-byte boundaries.  A warp owns 512 consecutive counts, read, cleared
 * and written 16 bytes per lane: with four words per thread and blocks of
 * 1,024 the 7 million cells of the full sweep took 80 to 120 us, waves of
 * blocks waiting at their barriers; this takes 14 (a million cells: the whole
 * scan 12 -> 8 us). */
constexpr int SCAN_COUNT_THREADS = 256;
constexpr int SCAN_COUNT_TRIPS = SCAN_TILE / (SCAN_COUNT_THREADS * 4);
template <bool NEXT>
__global__ void __launch_bounds__(SCAN_COUNT_THREADS) k_scan_counts(uint32_t* counts, uint32_t n,
                                                                    const uint32_t* __restrict__ block_sums,
                                                                    uint32_t* __restrict__ out) {
  __shared__ uint32_t warp_total[SCAN_COUNT_THREADS / 32], warp_before[SCAN_COUNT_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t base = blockIdx.x * SCAN_TILE + warp * (SCAN_COUNT_TRIPS * 128) + lane * 4;
  uint4 v[SCAN_COUNT_TRIPS];
#pragma unroll
  for (int q = 0; q < SCAN_COUNT_TRIPS; ++q) {
    const uint32_t c = base + q * 128;
    v[q] = make_uint4(0u, 0u, 0u, 0u);
    if (c + 4 <= n) {
      v[q] = *reinterpret_cast<const uint4*>(counts + c);
    } else {   /* the last few */
      if (c < n) v[q].x = counts[c];
      if (c + 1 < n) v[q].y = counts[c + 1];
      if (c + 2 < n) v[q].z = counts[c + 2];
    }
  }
  uint32_t before = 0;
  for (uint32_t b = threadIdx.x; b < blockIdx.x; b += SCAN_COUNT_THREADS) before += block_sums[b];
  /* exclusive prefix of each lane's words within the warp's segment */
  uint32_t e[SCAN_COUNT_TRIPS], carry = 0;
#pragma unroll
  for (int q = 0; q < SCAN_COUNT_TRIPS; ++q) {
    const uint32_t own = (v[q].x + v[q].y) + (v[q].z + v[q].w);
    uint32_t incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    e[q] = carry + incl - own;
    carry += __shfl_sync(0xffffffffu, incl, 31);
  }
  before = __reduce_add_sync(0xffffffffu, before);
  if (lane == 0) {
    warp_total[warp] = carry;
    warp_before[warp] = before;
  }
  __syncthreads();
  uint32_t offset = 0;
#pragma unroll
  for (int w = 0; w < SCAN_COUNT_THREADS / 32; ++w) offset += warp_before[w] + (w < warp ? warp_total[w] : 0u);
#pragma unroll
  for (int q = 0; q < SCAN_COUNT_TRIPS; ++q) {
    const uint32_t c = base + q * 128;
    const uint32_t e0 = offset + e[q], e1 = e0 + v[q].x, e2 = e1 + v[q].y, e3 = e2 + v[q].z;
    if (c + 4 <= n) {
      *reinterpret_cast<uint4*>(out + c) = make_uint4(e0, e1, e2, e3);
      if (NEXT) *reinterpret_cast<uint4*>(counts + c) = make_uint4(0u, 0u, 0u, 0u);
      if (NEXT && c + 4 == n) out[n] = e3 + v[q].w;
    } else if (c < n) {
      const uint32_t x[4] = {e0, e1, e2, e3};
      for (uint32_t k = 0; c + k < n; ++k) {
        out[c + k] = x[k];
        if (NEXT) counts[c + k] = 0u;
      }
      if (NEXT) out[n] = c + 1 == n ? e1 : (c + 2 == n ? e2 : e3);
    }
  }
}

/* VICSEK: the copy holds a heading's packed parts in place of (cos, sin). */
template <bool VICSEK>
__global__ void __launch_bounds__(SPP_BLOCK) k_scatter(DevState d) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  const uint32_t key = d.key[i];
  if (!spp_index_ok(d.ctl, key, d.n_keys)) return;
  uint32_t dst = d.cell_start[key] + d.rank[i];
  if (!spp_index_ok(d.ctl, dst, d.n)) return;
  float4 p = d.pos[i];
  if (VICSEK) {
    p.z = pack_parts(fx_parts(p.z));
    p.w = pack_parts(fx_parts(p.w));
  }
  d.pos_alt[dst] = p;
  d.theta_alt[dst] = d.theta[i];
  d.img_alt[dst] = d.img[i];
  d.id_alt[dst] = d.id[i];
}

/* Bound by its instruction stream (a thread per particle, about 15 candidates
 * for 5 neighbours).  At N = 1,048,576, ABP, unit density, 200 steps in: 87.6
 * us a launch when accepted neighbours were inserted in id order as they came
 * (each lane its own depth), 61 with them collected and put in order by a
 * network (build_particle_list); a whole rebuild 134 -> 98.  40 registers
 * for six blocks per SM; four or five are not faster.
 * Verlet list from the cell-ordered copy (alt), then the copy moves back
 * into the primary arrays. with_list == 0 only copies (no list).  The copy
 * always completes, even when some list overflows: the overflow only sets
 * the frozen flag, which stops the stage kernels until the host has grown
 * the list and rebuilt it. */
template <int LANES>
__global__ void __launch_bounds__(SPP_BLOCK, 6) k_build_list(SppConsts k, DevState d, int with_list) {
  __shared__ uint32_t slots[LIST_LOCAL][SPP_BLOCK];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t cnt = 0;
  if (i < d.n) {
    const float4 p = d.pos_alt[i];
    if (with_list) cnt = build_particle_list<LANES>(k, d, i, p, &slots[0][threadIdx.x], SPP_BLOCK);
    adopt_sorted_particle(d, i, p);
  }
  if (with_list) note_list_lengths(d, cnt);
  if (i == 0) atomicAdd(&d.ctl->n_rebuilds, 1u);
}

/* Lists longer than LIST_LOCAL, queued by k_build_list: one warp per list
 * (grid-stride over the queue). */
__global__ void __launch_bounds__(SPP_BLOCK) k_sort_long(SppConsts k, DevState d) {
  const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  const uint32_t total = d.ctl->long_n;
  for (uint32_t w = (uint32_t)warp; w < total; w += (uint32_t)nwarps) {
    sort_queued_list(k, d, d.long_q[w]);
  }
}

/* Unique pairs (by particle id) within r, through the cell list. */
__global__ void __launch_bounds__(SPP_BLOCK) k_pairs(SppConsts k, DevState d, float r2,
                                                     unsigned long long* counter, int32_t* pi,
                                                     int32_t* pj, long long cap) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  float4 p = d.pos[i];
  uint32_t idi = d.id[i];
  int cx, cy;
  cell_key(k, d, p.x, p.y, &cx, &cy);
  const int D = d.D;
  for (int oy = -1; oy <= 1; ++oy) {
    int ny = (cy + oy + D) % D;
    for (int ox = -1; ox <= 1; ++ox) {
      int nx = (cx + ox + D) % D;
      uint32_t kk = spp_morton((uint32_t)nx, (uint32_t)ny);
      uint32_t s0 = d.cell_start[kk], c = d.cell_count[kk];
      for (uint32_t j = s0; j < s0 + c; ++j) {
        uint32_t idj = d.id[j];
        if (idj <= idi) continue;
        float4 q = d.pos[j];
        float dx, dy;
        if (spp_sep(&k, p.x, p.y, q.x, q.y, &dx, &dy) < r2) {
          unsigned long long slot = atomicAdd(counter, 1ull);
          if ((long long)slot < cap) {
            pi[slot] = (int32_t)idi;
            pj[slot] = (int32_t)idj;
          }
        }
      }
    }
  }
}

__global__ void k_cells(SppConsts k, DevState d, int D, int rule, int32_t* cx, int32_t* cy) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  float4 p = d.pos[i];
  uint32_t id = d.id[i];
  cx[id] = spp_cell_coord(p.x, k.L, k.L2, D, rule);
  cy[id] = spp_cell_coord(p.y, k.L, k.L2, D, rule);
}

/* Places the uploaded state (particle-id order) and checks it: the smallest
 * index with a non-finite value and the smallest with a position outside
 * [-L, L) go to the control block, which the host reads before it accepts
 * the upload.  Invalid values stay bounded in what follows: cell
 * coordinates are clamped, and comparisons with NaN are false. */
__global__ void k_init_state(SppConsts k, DevState d, const float* __restrict__ x, const float* __restrict__ y,
                             const float* __restrict__ th, const int32_t* __restrict__ img_xy) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  const float xi = x[i], yi = y[i], ti = th[i];
  if (!isfinite(xi) || !isfinite(yi) || !isfinite(ti)) atomicMin(&d.ctl->bad_nonfinite, (uint32_t)i);
  else if (!k.closed && !(xi >= -k.L && xi < k.L && yi >= -k.L && yi < k.L))
    atomicMin(&d.ctl->bad_range, (uint32_t)i);  /* a closed box has no wrap to undo: any finite position */
  float s, c;
  spp_sincosf(ti, &s, &c);
  d.pos[i] = make_float4(xi, yi, c, s);
  d.theta[i] = ti;
  d.img[i] = img_xy ? make_int2(img_xy[i], img_xy[d.n + i]) : make_int2(0, 0);
  d.id[i] = (uint32_t)i;
}

__global__ void k_gather_state(DevState d, float* x, float* y, float* th, int32_t* img_xy) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  uint32_t id = d.id[i];
  float4 p = d.pos[i];
  x[id] = p.x;
  y[id] = p.y;
  th[id] = d.theta[i];
  const int2 g = d.img[i];
  img_xy[id] = g.x;
  img_xy[d.n + id] = g.y;
}

inline int blocks_for(int n, int b = SPP_BLOCK) { return (n + b - 1) / b; }

}  // namespace

void launch_bin_count(const SppConsts& k, const DevState& d, cudaStream_t s, int64_t* launches) {
  if (d.n == 0) return;
  k_bin_count<<<blocks_for(d.n), SPP_BLOCK, 0, s>>>(k, d);
  if (launches) *launches += 1;
}

void launch_scan_u32(uint32_t* counts, uint32_t n, uint32_t* block_tmp, uint32_t* out, cudaStream_t s,
                     int64_t* launches) {
  const uint32_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  k_scan_reduce<<<nb, SCAN_THREADS, 0, s>>>(counts, n, block_tmp);
  k_scan_counts<false><<<nb, SCAN_COUNT_THREADS, 0, s>>>(counts, n, block_tmp, out);
  if (launches) *launches += 2;
}

void launch_scan_counts(uint32_t* counts, uint32_t n, uint32_t* block_tmp, uint32_t* out, cudaStream_t s) {
  const uint32_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  k_scan_reduce<<<nb, SCAN_THREADS, 0, s>>>(counts, n, block_tmp);
  k_scan_counts<true><<<nb, SCAN_COUNT_THREADS, 0, s>>>(counts, n, block_tmp, out);
}

uint32_t scan_max_elements() { return (uint32_t)SCAN_TILE * (uint32_t)SCAN_TILE; }

void launch_scan(const DevState& d, cudaStream_t s, int64_t* launches) {
  launch_scan_u32(d.cell_count, d.n_keys, d.scan_tmp, d.cell_start, s, launches);
}

void launch_scatter(const DevState& d, bool vicsek, cudaStream_t s, int64_t* launches) {
  if (d.n == 0) return;
  if (vicsek) k_scatter<true><<<blocks_for(d.n), SPP_BLOCK, 0, s>>>(d);
  else k_scatter<false><<<blocks_for(d.n), SPP_BLOCK, 0, s>>>(d);
  if (launches) *launches += 1;
}

void launch_build_list(const SppConsts& k, const DevState& d, int with_list, cudaStream_t s,
                       int64_t* launches) {
  if (d.n == 0) return;
  if (with_list && k.lanes == SPP_GATHER_LANES)
    k_build_list<SPP_GATHER_LANES><<<blocks_for(d.n), SPP_BLOCK, 0, s>>>(k, d, with_list);
  else
    k_build_list<1><<<blocks_for(d.n), SPP_BLOCK, 0, s>>>(k, d, with_list);
  if (launches) *launches += 1;
  if (with_list) {
    /* 8 warps per block, 8 blocks per SM of a 152-SM part, looping over
     * the queue */
    int nb = (d.n + 7) / 8;
    if (nb > 1216) nb = 1216;
    k_sort_long<<<nb, SPP_BLOCK, 0, s>>>(k, d);
    if (launches) *launches += 1;
  }
}

void launch_pairs_count(const SppConsts& k, const DevState& d, float r2, unsigned long long* counter,
                        int32_t* pi, int32_t* pj, long long cap, cudaStream_t s) {
  if (d.n == 0) return;
  k_pairs<<<blocks_for(d.n), SPP_BLOCK, 0, s>>>(k, d, r2, counter, pi, pj, cap);
}

void launch_cells(const SppConsts& k, const DevState& d, int D, int rule, int32_t* cx, int32_t* cy,
                  cudaStream_t s) {
  if (d.n == 0) return;
  k_cells<<<blocks_for(d.n), SPP_BLOCK, 0, s>>>(k, d, D, rule, cx, cy);
}

void launch_init_state(const SppConsts& k, const DevState& d, const float* x, const float* y,
                       const float* th, const int32_t* img_xy, cudaStream_t s) {
  if (d.n == 0) return;
  k_init_state<<<blocks_for(d.n), SPP_BLOCK, 0, s>>>(k, d, x, y, th, img_xy);
}

void launch_gather_state(const SppConsts& k, const DevState& d, float* x, float* y, float* th,
                         int32_t* img_xy, cudaStream_t s) {
  (void)k;
  if (d.n == 0) return;
  k_gather_state<<<blocks_for(d.n), SPP_BLOCK, 0, s>>>(d, x, y, th, img_xy);
}
