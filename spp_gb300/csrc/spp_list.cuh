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

/* Accepted neighbours are collected as (id << 32 | slot) keys in a per-thread
 * array, insertion-sorted there (lists hold ~5 entries at unit density) and
 * written once; lists longer than the array fall back to sorting in place.
 * LIST_LOCAL keys are kept in shared memory per thread (a column of a
 * [LIST_LOCAL][threads] array: conflict-free); entries up to LIST_TAIL are
 * inserted in order in global memory, a list longer than that is finished
 * by sort_queued_list. */
#ifndef SPP_LIST_LOCAL
#define SPP_LIST_LOCAL 12
#endif
constexpr int LIST_LOCAL = SPP_LIST_LOCAL;
#ifndef SPP_LIST_TAIL
#define SPP_LIST_TAIL 16
#endif
constexpr int LIST_TAIL = SPP_LIST_TAIL;

/* spp_list_order with the lane count known at compile time */
template <int LANES>
__device__ __forceinline__ uint32_t list_order(uint32_t id) {
  return LANES == 1 ? id : ((id & 3u) << 30) | (id >> 2);
}

/* The list of the particle in slot i (position p) from the cell-ordered
 * copy: nbr, nn, nn_lanes and ref are written, a long list is queued.
 * col[q * stride], q < LIST_LOCAL, is the calling thread's column of shared
 * memory.  Returns the number of neighbours (which may exceed d.cap).
 *
 * The 3 x 3 cells are visited row by row with the three cells' ranges of a
 * row loaded together (three dependent round trips per particle instead of
 * nine) and walked as one sequence, two candidates per trip with both
 * candidates' positions and ids in flight; Morton keys built from per-axis
 * spreads, candidates read as (x, y) only, and the minimum image skipped for
 * particles far from the box edges (where it changes no separation within
 * the list radius, and a candidate across the edge is rejected either way).
 * Measured at the 1M workload 600 steps in (whole rebuild, us): 151.7 with
 * a cell-by-cell walk, 148.4 with rows one candidate per trip, 139.6 with
 * rows two per trip (40 registers; 141.9 when held to 32), 136.8 with the
 * ids loaded with the positions. */
template <int LANES>
__device__ __forceinline__ uint32_t build_particle_list(const SppConsts& k, const DevState& d, int i, float4 p,
                                                        unsigned long long* col, int stride) {
  uint32_t cnt = 0;
  unsigned long long lane_cnt = 0;   /* neighbours per id % 4, 16 bits each */
#define keys(q) col[(q) * stride]
  int cx, cy;
  cell_key(k, d, p.x, p.y, &cx, &cy);
  const int D = d.D;
  const uint32_t cap = (uint32_t)d.cap;
  /* one candidate j (cell-ordered slot) */
  auto visit = [&](uint32_t j, uint32_t idj, float dx, float dy, float d2) {
    if (d2 < k.rlist2) {
      const unsigned long long key =
          ((unsigned long long)list_order<LANES>(idj) << 32) | (unsigned long long)j;
      if (LANES > 1) lane_cnt += 1ull << (16 * (idj & 3u));
      if (cnt < (uint32_t)LIST_LOCAL) {
        /* the order words are unique, so comparing them orders the keys */
        const uint32_t ko = (uint32_t)(key >> 32);
        int pos = (int)cnt;
        while (pos > 0 && (uint32_t)(keys(pos - 1) >> 32) > ko) {
          keys(pos) = keys(pos - 1);
          --pos;
        }
        keys(pos) = key;
      } else if (cnt < cap && cnt < (uint32_t)LIST_TAIL) {
        /* a longer list: the first LIST_LOCAL keys are still local;
         * keep the next ones sorted in place in global memory */
        int pos = (int)cnt;
        while (pos > LIST_LOCAL) {
          const int32_t prev = d.nbr[(size_t)(pos - 1) * d.n + i];
          if (list_order<LANES>(d.id_alt[prev]) < (uint32_t)(key >> 32)) break;
          d.nbr[(size_t)pos * d.n + i] = prev;
          --pos;
        }
        if (pos == LIST_LOCAL && keys(LIST_LOCAL - 1) > key) {
          /* belongs among the local keys: swap with the local maximum */
          unsigned long long moved = keys(LIST_LOCAL - 1);
          int lp = LIST_LOCAL - 1;
          while (lp > 0 && keys(lp - 1) > key) {
            keys(lp) = keys(lp - 1);
            --lp;
          }
          keys(lp) = key;
          d.nbr[(size_t)pos * d.n + i] = (int32_t)(uint32_t)moved;
        } else {
          d.nbr[(size_t)pos * d.n + i] = (int32_t)j;
        }
      } else if (cnt < cap) {
        /* a long list: the rest is appended unsorted and k_sort_long
         * orders the whole list */
        d.nbr[(size_t)cnt * d.n + i] = (int32_t)j;
      }
      ++cnt;
    }
  };
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
    for (uint32_t t = 0; t < total; t += 2) {
      const uint32_t ja = slot_of(t);
      const uint32_t jb = t + 1 < total ? slot_of(t + 1) : ja;
      const float2 qa = reinterpret_cast<const float2*>(d.pos_alt)[2 * (size_t)ja];
      const float2 qb = reinterpret_cast<const float2*>(d.pos_alt)[2 * (size_t)jb];
      /* both ids with the positions: an accepted candidate's key does not
       * wait on a second load */
      const uint32_t ida = d.id_alt[ja], idb = d.id_alt[jb];
      float dxa, dya, dxb, dyb;
      const float d2a = wrap ? spp_pair_sep(&k, 1, p.x, p.y, qa.x, qa.y, &dxa, &dya)
                             : spp_pair_sep(&k, 0, p.x, p.y, qa.x, qa.y, &dxa, &dya);
      const float d2b = wrap ? spp_pair_sep(&k, 1, p.x, p.y, qb.x, qb.y, &dxb, &dyb)
                             : spp_pair_sep(&k, 0, p.x, p.y, qb.x, qb.y, &dxb, &dyb);
      if ((int)ja != i) visit(ja, ida, dxa, dya, d2a);
      if (t + 1 < total && (int)jb != i) visit(jb, idb, dxb, dyb, d2b);
    }
  }
  const uint32_t nloc = cnt < (uint32_t)LIST_LOCAL ? cnt : (uint32_t)LIST_LOCAL;
  const uint32_t nw = nloc < cap ? nloc : cap;
  for (uint32_t q = 0; q < nw; ++q) d.nbr[(size_t)q * d.n + i] = (int32_t)(uint32_t)keys(q);
  d.nn[i] = (int32_t)(cnt < cap ? cnt : cap);
  if (LANES > 1) d.nn_lanes[i] = lane_cnt;   /* meaningful when the list fits */
  if (cnt > (uint32_t)LIST_TAIL && cap > (uint32_t)LIST_TAIL)
    d.long_q[atomicAdd(&d.ctl->long_n, 1u)] = i;
  d.ref[i] = make_float2(p.x, p.y);
#undef keys
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

/* The list of particle i (m entries) insertion-sorted in place by one
 * thread: lists beyond 512 entries, which only extreme densities produce. */
__device__ __forceinline__ void insertion_sort_list(const SppConsts& k, const DevState& d, int i, int m) {
  for (int q = 1; q < m; ++q) {
    const int32_t j = d.nbr[(size_t)q * d.n + i];
    const uint32_t oj = spp_list_order(&k, d.id_alt[j]);
    int pos = q;
    while (pos > 0) {
      const int32_t prev = d.nbr[(size_t)(pos - 1) * d.n + i];
      if (spp_list_order(&k, d.id_alt[prev]) < oj) break;
      d.nbr[(size_t)pos * d.n + i] = prev;
      --pos;
    }
    d.nbr[(size_t)pos * d.n + i] = j;
  }
}

/* A queued list (longer than LIST_TAIL) put in order by the calling warp. */
__device__ __forceinline__ void sort_queued_list(const SppConsts& k, const DevState& d, int i) {
  if (!spp_index_ok(d.ctl, i, d.n)) return;
  const int m = d.nn[i];
  if (m <= 32) warp_sort_list<1>(k, d, i, m);
  else if (m <= 64) warp_sort_list<2>(k, d, i, m);
  else if (m <= 128) warp_sort_list<4>(k, d, i, m);
  else if (m <= 256) warp_sort_list<8>(k, d, i, m);
  else if (m <= 512) warp_sort_list<16>(k, d, i, m);
  else if ((threadIdx.x & 31) == 0) insertion_sort_list(k, d, i, m);
}

}  // namespace
#endif
