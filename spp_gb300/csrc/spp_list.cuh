/* spp_list.cuh -- device code of the neighbour-list build, shared by the
 * build kernels (kernels_cells.cu) and the resident step loop
 * (kernels_run.cu). */
#ifndef SPP_LIST_CUH
#define SPP_LIST_CUH
#include "spp_internal.cuh"

namespace {

__device__ __forceinline__ uint32_t cell_key(const SppConsts& k, const DevState& d, float x, float y,
                                             int* cx, int* cy) {
  *cx = spp_cell_coord(x, k.L, k.L2, d.D, SPP_BIN_GEOMETRIC);
  *cy = spp_cell_coord(y, k.L, k.L2, d.D, SPP_BIN_GEOMETRIC);
  return spp_morton((uint32_t)*cx, (uint32_t)*cy);
}

/* Exclusive prefix of v over the threads of the block (at most 32 warps),
 * and the block's total. */
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total = nullptr) {
  __shared__ uint32_t warp_sums[32];
  __shared__ uint32_t block_total;
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int nwarps = (int)(blockDim.x >> 5);
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < nwarps ? warp_sums[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    warp_sums[lane] = wi - w; /* exclusive prefix of the warp sums */
    if (lane == 31) block_total = wi;
  }
  __syncthreads();
  if (total) *total = block_total;
  return incl - v + warp_sums[warp];
}

/* Accepted neighbours are collected in visiting order, the slots of the first
 * LIST_LOCAL in the calling thread's column of shared memory (conflict-free),
 * the rest in the list itself.  A list that fits the column is put in order by
 * a sorting network in registers over (order word << 4 | place in the column)
 * and written once; a longer one is queued for sort_queued_list. */
constexpr int LIST_LOCAL = 16;
constexpr int LIST_TRIP = 2;   /* candidates in flight */

/* Batcher's odd-even merge sort (K. E. Batcher, Sorting networks and their
 * applications, 1968) of key[LO .. LO + N - 1]; entries from LIVE on hold the
 * largest key throughout, so comparisons with them are left out. */
template <int LIVE>
struct SortNetwork {
  template <int A, int B>
  static __device__ __forceinline__ void order(uint32_t* key) {
    if constexpr (B < LIVE) {
      const uint32_t lo = min(key[A], key[B]), hi = max(key[A], key[B]);
      key[A] = lo;
      key[B] = hi;
    }
  }
  template <int A, int END, int R, int STEP>
  static __device__ __forceinline__ void pairs(uint32_t* key) {
    if constexpr (A + R < END) {
      order<A, A + R>(key);
      pairs<A + STEP, END, R, STEP>(key);
    }
  }
  template <int LO, int N, int R>
  static __device__ __forceinline__ void merge(uint32_t* key) {
    if constexpr (2 * R < N) {
      merge<LO, N, 2 * R>(key);
      merge<LO + R, N, 2 * R>(key);
      pairs<LO + R, LO + N, R, 2 * R>(key);
    } else {
      order<LO, LO + R>(key);
    }
  }
  template <int LO, int N>
  static __device__ __forceinline__ void sort(uint32_t* key) {
    if constexpr (N > 1 && LO < LIVE) {
      sort<LO, N / 2>(key);
      sort<LO + N / 2, N / 2>(key);
      merge<LO, N, 1>(key);
    }
  }
};

/* The cnt <= LIVE collected slots of a thread (col[q * stride]) into its list
 * in order; returns the neighbours per id % 4 for LANES > 1. */
template <int LANES, int LIVE>
__device__ __forceinline__ unsigned long long write_sorted_list(const DevState& d, int i, uint32_t cnt,
                                                                const uint32_t* col, int stride) {
  unsigned long long lane_cnt = 0;
  uint32_t key[LIVE <= 8 ? 8 : 16];
#pragma unroll
  for (int q = 0; q < (LIVE <= 8 ? 8 : 16); ++q) {
    key[q] = 0xffffffffu;
    if (q < LIVE && (uint32_t)q < cnt) {
      const uint32_t id = d.id_alt[col[q * stride]];
      if (LANES > 1) lane_cnt += 1ull << (16 * (id & 3u));
      /* ids below 2^28, so the order word fits 28 bits */
      key[q] = (LANES == 1 ? id : ((id & 3u) << 26) | (id >> 2)) << 4 | (uint32_t)q;
    }
  }
  SortNetwork<LIVE>::template sort<0, (LIVE <= 8 ? 8 : 16)>(key);
#pragma unroll
  for (int q = 0; q < LIVE; ++q)
    if ((uint32_t)q < cnt) d.nbr[(size_t)q * d.n + i] = (int32_t)col[(key[q] & 15u) * stride];
  return lane_cnt;
}

/* The list of the particle in slot i (position p) from the cell-ordered
 * copy: nbr, nn, nn_lanes and ref are written, a long list is queued.
 * col[q * stride], q < LIST_LOCAL, is the calling thread's column of shared
 * memory.  Returns the number of neighbours (which may exceed d.cap).
 *
 * The 3 x 3 cells are visited row by row with the three cells' ranges of a
 * row loaded together (three dependent round trips per particle instead of
 * nine) and walked as one sequence, two candidates per trip with both
 * candidates' positions in flight; Morton keys built from per-axis
 * spreads, candidates read as (x, y) only, and the minimum image skipped for
 * particles far from the box edges (where it changes no separation within
 * the list radius, and a candidate across the edge is rejected either way).
 * Measured at the 1M workload 600 steps in (whole rebuild, us): 151.7 with
 * a cell-by-cell walk, 148.4 with rows one candidate per trip, 139.6 with
 * rows two per trip (40 registers; 141.9 when held to 32).  The order comes
 * at the end, all lanes in step, instead of by insertion as candidates are
 * accepted, and a candidate is stored whether taken or not (98 against 101 with
 * a branch): 134 -> 98 200 steps in; 50 steps of resident runs of 16,384
 * particles 1,254 -> 1,120 us (one candidate per trip 1,170), of 163,840 beads
 * 1,240 -> 1,107. */
template <int LANES>
__device__ __forceinline__ uint32_t build_particle_list(const SppConsts& k, const DevState& d, int i, float4 p,
                                                        uint32_t* col, int stride) {
  uint32_t cnt = 0;
  int cx, cy;
  cell_key(k, d, p.x, p.y, &cx, &cy);
  const int D = d.D;
  const uint32_t cap = (uint32_t)d.cap;
  const int wrap = !(k.closed || (fabsf(p.x) < k.interior && fabsf(p.y) < k.interior));
  uint32_t mx[3];
#pragma unroll
  for (int o = 0; o < 3; ++o) {
    int nx = cx + o - 1;
    nx = nx < 0 ? nx + D : (nx >= D ? nx - D : nx);
    mx[o] = spp_morton_spread((uint32_t)nx);
  }
  for (int oy = -1; oy <= 1; ++oy) {
    int ny = cy + oy;
    ny = ny < 0 ? ny + D : (ny >= D ? ny - D : ny);
    const uint32_t my = spp_morton_spread((uint32_t)ny) << 1;
    uint32_t s0[3], c[3];
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      const uint32_t kk = mx[o] | my;
      s0[o] = 0u;
      c[o] = 0u;
      if (!spp_index_ok(d.ctl, kk, d.n_keys)) continue;
      s0[o] = d.cell_start[kk];
      c[o] = d.cell_count[kk];
      if (!spp_index_ok(d.ctl, (long long)s0[o] + c[o], (long long)d.n + 1)) c[o] = 0u;
    }
    /* the row's three ranges as one sequence, two candidates per trip
     * with both loads in flight */
    const uint32_t c01 = c[0] + c[1], total = c01 + c[2];
    auto slot_of = [&](uint32_t t) {
      return t < c[0] ? s0[0] + t : (t < c01 ? s0[1] + (t - c[0]) : s0[2] + (t - c01));
    };
    for (uint32_t t = 0; t < total; t += LIST_TRIP) {
      uint32_t j[LIST_TRIP];
      float2 q[LIST_TRIP];
#pragma unroll
      for (int u = 0; u < LIST_TRIP; ++u) {
        j[u] = t + u < total ? slot_of(t + u) : (uint32_t)i;
        q[u] = reinterpret_cast<const float2*>(d.pos_alt)[2 * (size_t)j[u]];
      }
      float d2[LIST_TRIP];
#pragma unroll
      for (int u = 0; u < LIST_TRIP; ++u) {
        float dx, dy;
        d2[u] = wrap ? spp_pair_sep(&k, 1, p.x, p.y, q[u].x, q[u].y, &dx, &dy)
                     : spp_pair_sep(&k, 0, p.x, p.y, q[u].x, q[u].y, &dx, &dy);
      }
#pragma unroll
      for (int u = 0; u < LIST_TRIP; ++u) {
        const bool ok = d2[u] < k.rlist2 && (int)j[u] != i;
        if (cnt < (uint32_t)LIST_LOCAL) col[cnt * stride] = j[u];   /* taken or overwritten: no lane waits */
        else if (ok && cnt < cap) d.nbr[(size_t)cnt * d.n + i] = (int32_t)j[u];
        cnt += ok;
      }
    }
  }
  unsigned long long lane_cnt = 0;   /* neighbours per id % 4, 16 bits each */
  const bool queued = cnt > (uint32_t)LIST_LOCAL || d.n > 1 << 28;
  const uint32_t in_order = queued || cnt > cap ? 0u : cnt;
  const uint32_t longest = __reduce_max_sync(__activemask(), in_order);
  if (longest > 12u) lane_cnt = write_sorted_list<LANES, 16>(d, i, in_order, col, stride);
  else if (longest > 8u) lane_cnt = write_sorted_list<LANES, 12>(d, i, in_order, col, stride);
  else lane_cnt = write_sorted_list<LANES, 8>(d, i, in_order, col, stride);
  if (in_order < cnt) {   /* the queue's, or too long for the list (the run stops and grows it) */
    const uint32_t held = cnt < cap ? cnt : cap;
    for (uint32_t q = 0; q < held && q < (uint32_t)LIST_LOCAL; ++q) d.nbr[(size_t)q * d.n + i] = (int32_t)col[q * stride];
    if (LANES > 1)
      for (uint32_t q = 0; q < held; ++q) lane_cnt += 1ull << (16 * (d.id_alt[d.nbr[(size_t)q * d.n + i]] & 3u));
    if (queued) d.long_q[atomicAdd(&d.ctl->long_n, 1u)] = i;
  }
  d.nn[i] = (int32_t)(cnt < cap ? cnt : cap);
  if (LANES > 1) d.nn_lanes[i] = lane_cnt;   /* meaningful when the list fits */
  d.ref[i] = make_float2(p.x, p.y);
  return cnt;
}

/* The cell-ordered copy's particle of slot i (position p) into the primary
 * arrays. */
__device__ __forceinline__ void adopt_sorted_particle(const DevState& d, int i, float4 p) {
  d.pos[i] = p;
  d.theta[i] = d.theta_alt[i];
  d.img[i] = d.img_alt[i];
  const uint32_t id = d.id_alt[i];
  d.id[i] = id;
  if (d.inv) d.inv[id] = (uint32_t)i;
}

/* The longest list of the warp's particles; an overflow freezes the system
 * (all 32 lanes call). */
__device__ __forceinline__ void note_list_lengths(const DevState& d, uint32_t cnt) {
  const uint32_t m = __reduce_max_sync(0xffffffffu, cnt);
  if ((threadIdx.x & 31) == 0 && m > 0) {
    atomicMax(&d.ctl->max_nn, m);
    if (m > (uint32_t)d.cap) {
      atomicMax(&d.ctl->list_need, m);
      atomicExch(&d.ctl->frozen, 1u);
    }
  }
}

/* Sorts the list of particle i (m entries, m <= 32 R) by (id, slot): one
 * warp, R keys per lane, element e = r * 32 + lane, a bitonic network
 * (partners across lanes by shuffle, across r in registers).  Ids are
 * unique, so the order is the one the insertion sort of short lists gives. */
template <int R>
__device__ __forceinline__ void warp_sort_list(const SppConsts& k, const DevState& d, int i, int m) {
  const int lane = threadIdx.x & 31;
  unsigned long long key[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int q = r * 32 + lane;
    if (q < m) {
      int32_t j = d.nbr[(size_t)q * d.n + i];
      if (!spp_index_ok(d.ctl, j, d.n)) j = i;
      key[r] = ((unsigned long long)spp_list_order(&k, d.id_alt[j]) << 32) | (unsigned long long)(uint32_t)j;
    } else {
      key[r] = ~0ull;
    }
  }
#pragma unroll
  for (int size = 2; size <= 32 * R; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (stride >= 32) {
        const int rs = stride >> 5;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int rp = r ^ rs;
          if (rp > r) {
            const bool up = ((r * 32 + lane) & size) == 0;
            const unsigned long long a = key[r], b = key[rp];
            if (up ? (a > b) : (a < b)) {
              key[r] = b;
              key[rp] = a;
            }
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const unsigned long long other = __shfl_xor_sync(0xffffffffu, key[r], stride);
          const bool up = ((r * 32 + lane) & size) == 0;
          const bool lower = (lane & stride) == 0;
          const bool keep_min = (up == lower);
          const unsigned long long lo = key[r] < other ? key[r] : other;
          const unsigned long long hi = key[r] < other ? other : key[r];
          key[r] = keep_min ? lo : hi;
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int q = r * 32 + lane;
    if (q < m) d.nbr[(size_t)q * d.n + i] = (int32_t)(uint32_t)key[r];
  }
}

/* The list of particle i (m entries) sorted in place by the calling warp:
 * lists beyond 512 entries, which only clumps produce.  Batcher's bitonic
 * sorter for any m: a merge of runs compares mirrored places first, then
 * places a stride apart, always ascending, so the places from m on, which
 * hold the largest keys, never exchange.  A resident run does this between
 * grid barriers that give up after seconds, so the time has to be bounded: a
 * list of 5,000 takes 91 passes of 128 comparisons per lane (an insertion by
 * one lane took 6 million dependent loads, some seconds). */
__device__ __forceinline__ void sort_list_in_place(const SppConsts& k, const DevState& d, int i, int m) {
  const int lane = threadIdx.x & 31;
  auto exchange = [&](int lo, int hi) {
    if (hi >= m) return;
    int32_t* const a = d.nbr + (size_t)lo * d.n + i;
    int32_t* const b = d.nbr + (size_t)hi * d.n + i;
    const int32_t ja = *a, jb = *b;
    if (!spp_index_ok(d.ctl, ja, d.n) || !spp_index_ok(d.ctl, jb, d.n)) return;
    if (spp_list_order(&k, d.id_alt[ja]) > spp_list_order(&k, d.id_alt[jb])) {
      *a = jb;
      *b = ja;
    }
  };
  int size = 2;
  while (size < m) size <<= 1;
  for (int run = 2; run <= size; run <<= 1) {
    for (int e = lane; e < size / 2; e += 32) {
      const int at = e / (run / 2) * run, o = e % (run / 2);
      exchange(at + o, at + run - 1 - o);
    }
    __syncwarp();
    for (int stride = run >> 2; stride > 0; stride >>= 1) {
      for (int e = lane; e < size / 2; e += 32) {
        const int lo = 2 * e - (e & (stride - 1));
        exchange(lo, lo + stride);
      }
      __syncwarp();
    }
  }
}

/* A queued list (longer than LIST_LOCAL) put in order by the calling warp. */
__device__ __forceinline__ void sort_queued_list(const SppConsts& k, const DevState& d, int i) {
  if (!spp_index_ok(d.ctl, i, d.n)) return;
  const int m = d.nn[i];
  if (m <= 32) warp_sort_list<1>(k, d, i, m);
  else if (m <= 64) warp_sort_list<2>(k, d, i, m);
  else if (m <= 128) warp_sort_list<4>(k, d, i, m);
  else if (m <= 256) warp_sort_list<8>(k, d, i, m);
  else if (m <= 512) warp_sort_list<16>(k, d, i, m);
  else sort_list_in_place(k, d, i, m);
}

}  // namespace
#endif
