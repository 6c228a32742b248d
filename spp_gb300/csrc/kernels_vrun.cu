/*
 * kernels_vrun.cu -- resident runs of the discrete Vicsek models: many steps
 * in one cooperative launch, one grid barrier per step, on sm_103a.
 *
 * k_vrun advances VicsekParticle{,2}::Interact/Move (shared/particle.h:
 * 145-247) and the arg-sum rule with every particle owned by LANES threads
 * for the whole launch.  Cells are buckets of fixed capacity in global
 * memory: a particle that has moved takes a place in its new cell by one
 * atomicAdd and writes its state there, in the buckets the next step reads;
 * the barrier after it orders the writes before those reads.  So a step
 * needs no counting pass, scan or scatter, and a thread can ask for its
 * cells' counts and first entries in one round of loads.  The sums are exact
 * fixed point: the places' arrival order does not matter, and the result is
 * that of the multi-kernel step (k_bin_count / scan / k_scatter /
 * k_vicsek_step) bit for bit.
 *
 * Every RUN_SORT_STEPS steps, over calls, the particles change hands in cell
 * order (a scan of the counts, a scatter, three barriers), so that a warp's
 * threads read the same cells.  A step in which some cell holds more than the bucket's
 * capacity (flocks) does the same and takes its candidates from the sorted
 * copy; the run stays in this kernel.
 *
 * Why: a step of six dependent kernels is bound by their latency.  Measured
 * (one GB300, vector rule, unit density, eta = 0.3, flocking; us per step):
 * N = 4,096 30.9 -> 6.5 (12.8 in one cluster of 16 CTAs, the former path of
 * systems up to 16,384); 16,384 35.4 -> 8.0; 50,001 42.5 -> 13.6; 175,104
 * 59.0 -> 27.8.  What bounds it now: small systems the chain barrier (1.1 us)
 * -> counts and first candidates -> the rest of the candidates -> update ->
 * place in the cell (an atomic's round trip) -> stores visible; large ones
 * the candidate walk, whose length is the warp's longest.  A second copy of
 * the walk without images, for warps away from the box edges, and packed
 * headings that take two additions a term: 7.5 -> 6.9 us at N = 4,096, 25.0 ->
 * 21.9 at 50,001 and density 2, 52.5 -> 44.3 at 175,000 (with push 197 -> 146).
 * Candidates in flight, vector rule: 3 / 4 / 6 take 7.3 / 6.9 / 6.6, 24.1 /
 * 21.9 / 20.0 and 49.6 / 44.3 / 39.8; the other rules, whose terms need the
 * registers: angles at 50,001 15.9 / 15.7 / 16.7, push 59 / 56 / 55.
 * Without the sorts N = 50,001 took 28.4 (17.0 with them at the time), with
 * one every 8 steps as long as with one every 16.  Counted over calls (calls of
 * 16 steps at N = 4,097 / 50,001 / 120,001: 6.6 / 16.7 / 25.3 us when every call
 * counted for itself, 6.1 / 13.9 / 22.4 now; calls of 100: 5.6 / 13.4 / 21.8).
 */
#include "spp_internal.cuh"
#include "spp_grid.cuh"
#include "spp_pack.cuh"
#include <algorithm>
#include <type_traits>

namespace {

__host__ __device__ constexpr int vrun_threads(int per_sm) { return per_sm == 1 ? 640 : 576; }

/* A bucket entry: position, and the packed parts of cos and sin. */
__device__ __forceinline__ float pack_fx(float v) { return pack_parts(fx_parts(v)); }

/* The sums a particle receives. */
struct VrunAcc {
  PackedSum cx, cy;   /* headings of the aligning neighbours */
  SppAcc a;           /* count, angles (ax, ay: the push terms) */
};

/* One candidate (entry q, heading thj for the angle rule); the terms of
 * spp_pair_vicsek.  WRAP: some image may be nearer. */
template <int MODEL, bool WRAP>
__device__ __forceinline__ void vrun_pair(const SppConsts& k, VrunAcc* acc, float4 p, float4 q, float thj, bool self) {
  float dx, dy;
  const float d2 = spp_pair_sep(&k, WRAP, p.x, p.y, q.x, q.y, &dx, &dy);
  if (!(d2 < k.ral2)) return;
  if (MODEL != SPP_MODEL_VICSEK && self) return;   /* the vector sum counts the particle itself */
  acc->a.cnt += 1;
  if (MODEL == SPP_MODEL_VICSEK_REF_ANGLE) {
    spp_fx_add_guarded(&acc->a.at, thj, &acc->a.ovf);
    return;
  }
  packed_add(&acc->cx, q.z);
  packed_add(&acc->cy, q.w);
  if (MODEL == SPP_MODEL_VICSEK_REF_VECTOR && d2 < k.rpush2 && d2 > 0.0f) spp_push_vicsek(&k, &acc->a, dx, dy, d2);
}

/* Counts are kept for three steps, buckets for two: step t reads count
 * t % 3 and bucket t % 2, fills (t + 1) % 3 and (t + 1) % 2, and clears count
 * (t + 2) % 3, which every block has finished reading before the barrier of
 * step t - 1.  full[c]: some cell of count c overflowed its bucket.
 * The last step fills nothing, so a launch leaves two clean counts, and the
 * next goes on with them (t % 3 stands for (t + *vb.phase) % 3): it clears the
 * third in its first step, and the one barrier after the particles are in
 * their cells is all that it pays to start.  us per call of one step, counts
 * cleared behind a barrier at the start and one more barrier at the end / now:
 * vector rule N = 1 10.5 / 8.7, 300 10.8 / 8.7, 4,096 14.0 / 10.8, 50,001 22.8 / 18.0
 * (one cluster of 16 CTAs took 8.7, 10.7 and 17.9 for the first three). */
template <int MODEL, int LANES, int PER_SM>
__global__ void __launch_bounds__(vrun_threads(PER_SM), PER_SM)
    k_vrun(const __grid_constant__ SppConsts k, const __grid_constant__ DevState d, const __grid_constant__ VrunBufs vb,
           int nsteps, int first, int every, unsigned long long* sums) {
  constexpr bool ANGLE = MODEL == SPP_MODEL_VICSEK_REF_ANGLE;
  constexpr int NC = (9 + LANES - 1) / LANES;   /* cells per lane */
  constexpr int AT_ONCE = 3;                    /* cells whose loads are issued together */
  constexpr int DEPTH = MODEL == SPP_MODEL_VICSEK ? 6 : 4;   /* candidates whose loads are issued together */
  __shared__ unsigned s_word;
  __shared__ unsigned long long s_sum[2];
  const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31;
  const int gthreads = gridDim.x * T, gtid = blockIdx.x * T + tid;
  Ctl* const ctl = d.ctl;
  const int n = d.n, D = d.D, K = vb.cap;
  const int i = gtid / LANES;
  const int lane_r = LANES == 1 ? 0 : tid % LANES;
  const bool inb = i < n;
  const bool head = inb && lane_r == 0;
  if (ctl->run_timeout) return;   /* the same for every block */
  const bool dirty = *vb.dirty != 0u;
  /* counts and flags of the step at hand, of the next, and those to be cleared
   * (in registers, rotated: indices cost the angle rule 3%) */
  const uint32_t phase = *vb.phase % 3u;
  uint32_t *cnow = vb.count[phase], *cnext = vb.count[(phase + 1u) % 3u], *cold = vb.count[(phase + 2u) % 3u];
  uint32_t *fnow = vb.full + phase, *fnext = vb.full + (phase + 1u) % 3u, *fold = vb.full + (phase + 2u) % 3u;
  uint32_t step = ctl->step, sorted = ctl->run_sorted;
  unsigned target = 0;
  auto barrier = [&]() -> bool {
    target += gridDim.x;
    __syncthreads();
    if (tid == 0) {
      grid_arrive(ctl);
      s_word = grid_wait(ctl, target);
      if (s_word == 0u) *vb.dirty = 1u;
    }
    __syncthreads();
    return s_word != 0u;
  };

  float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float th = 0.0f;
  uint32_t pid = 0u;
  if (inb) {
    p = d.pos[i];
    th = d.theta[i];
    pid = d.id[i];
  }
  int cx = 0, cy = 0;
  uint32_t rank = 0u;
  /* the particle's place among the cells of step t */
  auto insert = [&](int t, uint32_t* counts, uint32_t* flag) {
    if (head) {
      cx = spp_cell_coord(p.x, k.L, k.L2, D, SPP_BIN_GEOMETRIC);
      cy = spp_cell_coord(p.y, k.L, k.L2, D, SPP_BIN_GEOMETRIC);
      const uint32_t cell = (uint32_t)cy * (uint32_t)D + (uint32_t)cx;
      rank = atomicAdd(counts + cell, 1u);
      if (rank < (uint32_t)K) {
        const size_t at = (size_t)cell * K + rank;
        vb.bucket[t & 1][at] = make_float4(p.x, p.y, pack_fx(p.z), pack_fx(p.w));
        if (ANGLE) vb.bucket_th[t & 1][at] = th;
      } else {
        *flag = 1u;
      }
    }
    if (LANES > 1) {
      const int src = lane & ~(LANES - 1);
      p.x = __shfl_sync(0xffffffffu, p.x, src);
      p.y = __shfl_sync(0xffffffffu, p.y, src);
      cx = __shfl_sync(0xffffffffu, cx, src);
      cy = __shfl_sync(0xffffffffu, cy, src);
      rank = __shfl_sync(0xffffffffu, rank, src);
    }
  };
  /* the block's part of the heading sums of k_polarization: exact, whatever
   * the order */
  auto frame_sums = [&]() {
    long long sx = 0, sy = 0;
    if (head) {
      spp_fx hx = {0, 0}, hy = {0, 0};
      spp_fx_add(&hx, p.z);
      spp_fx_add(&hy, p.w);
      sx = spp_fx_units(hx);
      sy = spp_fx_units(hy);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sx += __shfl_down_sync(0xffffffffu, sx, o);
      sy += __shfl_down_sync(0xffffffffu, sy, o);
    }
    if (lane == 0) {
      atomicAdd(&s_sum[0], (unsigned long long)sx);
      atomicAdd(&s_sum[1], (unsigned long long)sy);
    }
  };
  if (tid < 2) s_sum[tid] = 0ull;
  if (dirty) {   /* the same for every block: written behind a barrier or by an earlier launch */
    for (uint32_t c = gtid; c < vb.cells; c += gthreads) vb.count[0][c] = vb.count[1][c] = vb.count[2][c] = 0u;
    if (gtid < 3) vb.full[gtid] = 0u;
    if (!barrier()) return;
    if (gtid == 0) *vb.dirty = 0u;
  }
  insert(0, cnow, fnow);
  uint32_t word = head ? spp_draw_k(&k, pid, step, SPP_RNG_VICSEK).v[0] : 0u;
  if (!barrier()) return;

  int to_frame = first;
  for (int t = 0;; ++t, ++step) {
    {
      for (uint32_t c = gtid; c < vb.cells; c += gthreads) cold[c] = 0u;
      if (gtid == 0) *fold = 0u;
    }
    const uint32_t* const count = cnow;
    const unsigned full = *(volatile const unsigned*)fnow;   /* the same for every thread of the grid */
    if (full || spp_sort_due(step, sorted)) {
      sorted = step;
      /* the particles change hands in cell order, so that a warp's threads
       * read the same cells; with a full bucket the step's candidates come
       * from this copy */
      if (!grid_scan(count, d.cell_start, vb.cells, d.run_sums, barrier)) return;
      if (!barrier()) return;
      if (head) {
        const uint32_t to = d.cell_start[(uint32_t)cy * (uint32_t)D + (uint32_t)cx] + rank;
        if (spp_index_ok(ctl, to, n)) {
          d.pos_alt[to] = make_float4(p.x, p.y, pack_fx(p.z), pack_fx(p.w));
          d.theta_alt[to] = th;
          d.img_alt[to] = d.img[i];
          d.id_alt[to] = pid;
        }
      }
      if (!barrier()) return;
      if (inb) {
        p = d.pos_alt[i];
        cx = spp_cell_coord(p.x, k.L, k.L2, D, SPP_BIN_GEOMETRIC);
        cy = spp_cell_coord(p.y, k.L, k.L2, D, SPP_BIN_GEOMETRIC);
        rank = (uint32_t)i - d.cell_start[(uint32_t)cy * (uint32_t)D + (uint32_t)cx];
      }
      if (head) {
        th = d.theta_alt[i];
        pid = d.id_alt[i];
        spp_sincosf(th, &p.w, &p.z);   /* (cos, sin) theta, as every update leaves them */
        d.img[i] = d.img_alt[i];
        word = spp_draw_k(&k, pid, step, SPP_RNG_VICSEK).v[0];
      }
    }
    const float4* const cand = full ? d.pos_alt : vb.bucket[t & 1];
    const float* const cand_th = full ? d.theta_alt : vb.bucket_th[t & 1];
    VrunAcc acc;
    acc.cx = acc.cy = {0, 0};
    spp_acc_zero(&acc.a);
    auto cell_of = [&](int c9) -> uint32_t {
      int ny = cy + c9 / 3 - 1, nx = cx + c9 % 3 - 1;
      ny = ny < 0 ? ny + D : (ny >= D ? ny - D : ny);
      nx = nx < 0 ? nx + D : (nx >= D ? nx - D : nx);
      return (uint32_t)ny * (uint32_t)D + (uint32_t)nx;
    };
    auto walk = [&](auto wrapped) {
      constexpr bool WRAP = decltype(wrapped)::value;
#pragma unroll 1
      for (int m0 = 0; inb && m0 < NC; m0 += AT_ONCE) {
        /* a cell's candidates: cnt of them from base on; the first of each is
         * asked for before the count is known (a place not taken holds an
         * older state, not used) */
        uint32_t cnt[AT_ONCE], base[AT_ONCE];
        float4 q[AT_ONCE];
        float qt[AT_ONCE];
#pragma unroll
        for (int m = 0; m < AT_ONCE; ++m) {
          const int c9 = lane_r + LANES * (m0 + m);
          const bool is = m0 + m < NC && c9 < 9;
          const uint32_t cell = cell_of(is ? c9 : 4);
          cnt[m] = is ? count[cell] : 0u;
          base[m] = full ? min(d.cell_start[cell], (uint32_t)n - 1u) : cell * (uint32_t)K;
          q[m] = cand[base[m]];
          qt[m] = ANGLE ? cand_th[base[m]] : 0.0f;
        }
#pragma unroll
        for (int m = 0; m < AT_ONCE; ++m)
          if (cnt[m] > 0u)
            vrun_pair<MODEL, WRAP>(k, &acc, p, q[m], qt[m], lane_r + LANES * (m0 + m) == 4 && rank == 0u);
        /* the rest of the cells as one sequence, DEPTH at a time: lanes differ
         * only in its length */
        int l[AT_ONCE + 1];
        l[0] = 0;
#pragma unroll
        for (int m = 0; m < AT_ONCE; ++m) l[m + 1] = l[m] + max((int)cnt[m] - 1, 0);
        for (int s = 0; s < l[AT_ONCE]; s += DEPTH) {
          float4 qs[DEPTH];
          float ts[DEPTH];
          bool self[DEPTH];
#pragma unroll
          for (int u = 0; u < DEPTH; ++u) {
            const int v = min(s + u, l[AT_ONCE] - 1);
            uint32_t at = base[0];
            int off = -1, c9 = lane_r + LANES * m0;
#pragma unroll
            for (int w = 1; w < AT_ONCE; ++w)
              if (v >= l[w]) {
                at = base[w];
                off = l[w] - 1;
                c9 = lane_r + LANES * (m0 + w);
              }
            const uint32_t e = (uint32_t)(v - off);
            qs[u] = cand[at + e];
            ts[u] = ANGLE ? cand_th[at + e] : 0.0f;
            self[u] = c9 == 4 && e == rank;
          }
#pragma unroll
          for (int u = 0; u < DEPTH; ++u)
            if (s + u < l[AT_ONCE]) vrun_pair<MODEL, WRAP>(k, &acc, p, qs[u], ts[u], self[u]);
        }
      }
    };
    /* a candidate of an interior cell is nearest as it is (or two cells away,
     * beyond every cutoff), and a closed box has no images */
    const int plain = !inb || k.closed || (cx >= 1 && cx <= D - 2 && cy >= 1 && cy <= D - 2);
    if (__all_sync(0xffffffffu, plain)) walk(std::false_type{});
    else walk(std::true_type{});
    SppAcc& a = acc.a;
    if (!ANGLE) {
      const spp_fx fx = packed_value(acc.cx, a.cnt), fy = packed_value(acc.cy, a.cnt);
      a.ax.hi += fx.hi;
      a.ax.lo += fx.lo;
      a.ay.hi += fy.hi;
      a.ay.lo += fy.lo;
    }
    if (LANES > 1) {
#pragma unroll
      for (int o = 1; o < LANES; o <<= 1) {
        if (!ANGLE) {
          a.ax.hi += __shfl_xor_sync(0xffffffffu, a.ax.hi, o);
          a.ax.lo += __shfl_xor_sync(0xffffffffu, a.ax.lo, o);
          a.ay.hi += __shfl_xor_sync(0xffffffffu, a.ay.hi, o);
          a.ay.lo += __shfl_xor_sync(0xffffffffu, a.ay.lo, o);
        } else {
          a.at.hi += __shfl_xor_sync(0xffffffffu, a.at.hi, o);
          a.at.lo += __shfl_xor_sync(0xffffffffu, a.at.lo, o);
        }
        a.cnt += __shfl_xor_sync(0xffffffffu, a.cnt, o);
        a.ovf |= __shfl_xor_sync(0xffffffffu, a.ovf, o);
      }
    }
    if (head) {
      if (ANGLE && k.closed) spp_vicsek_walls(&k, &a, p.x, p.y, th);
      if (a.ovf) atomicOr(&ctl->fx_overflow, 1u);
      float x, y, nt, c, s;
      int gx = 0, gy = 0;
      spp_vicsek_update(&k, &a, p.x, p.y, th, p.z, p.w, word, &x, &y, &nt, &c, &s, &gx, &gy);
      p = make_float4(x, y, c, s);
      th = nt;
      if (gx | gy) {   /* only this thread touches the particle's counters */
        const int2 g = d.img[i];
        d.img[i] = make_int2(g.x + gx, g.y + gy);
      }
    }
    const bool frame = every > 0 && --to_frame == 0;
    if (t + 1 == nsteps) {   /* nothing of this launch follows */
      if (frame) {
        frame_sums();
        __syncthreads();
        if (tid == 0) {
          atomicAdd(sums, s_sum[0]);
          atomicAdd(sums + 1, s_sum[1]);
        }
      }
      break;
    }
    insert(t + 1, cnext, fnext);
    if (frame) frame_sums();
    target += gridDim.x;
    __syncthreads();
    if (tid == 0) {
      grid_arrive(ctl);
      if (frame) {
        atomicAdd(sums, s_sum[0]);
        atomicAdd(sums + 1, s_sum[1]);
        s_sum[0] = s_sum[1] = 0ull;
      }
    }
    if (frame) {
      sums += 2;
      to_frame = every;
    }
    {
      uint32_t* const c = cnow;
      cnow = cnext;
      cnext = cold;
      cold = c;
      uint32_t* const f = fnow;
      fnow = fnext;
      fnext = fold;
      fold = f;
    }
    /* the next step's noise while the other blocks arrive */
    if (head) word = spp_draw_k(&k, pid, step + 1u, SPP_RNG_VICSEK).v[0];
    if (tid == 0) {
      s_word = grid_wait(ctl, target);
      if (s_word == 0u) *vb.dirty = 1u;
    }
    __syncthreads();
    if (s_word == 0u) return;
  }

  if (head) {
    d.pos[i] = p;
    d.theta[i] = th;
    d.id[i] = pid;
  }
  if (tid == 0) {
    if (blockIdx.x == 0) {
      ctl->step = step + 1u;
      ctl->run_sorted = sorted;
      *vb.phase = (phase + (uint32_t)nsteps) % 3u;
      ctl->need_rebuild = 0u;
    }
    /* the last block to leave clears the barrier for the next launch */
    __threadfence();
    if (atomicAdd(&ctl->run_exit, 1u) == gridDim.x - 1) {
      ctl->run_bar = 0u;
      ctl->run_exit = 0u;
    }
  }
}

typedef void (*VrunKernel)(SppConsts, DevState, VrunBufs, int, int, int, unsigned long long*);

template <int MODEL>
VrunKernel vrun_kernel_for(int lanes, int per_sm) {
  if (lanes == 4) return per_sm == 1 ? (VrunKernel)k_vrun<MODEL, 4, 1> : (VrunKernel)k_vrun<MODEL, 4, 2>;
  if (lanes == 2) return per_sm == 1 ? (VrunKernel)k_vrun<MODEL, 2, 1> : (VrunKernel)k_vrun<MODEL, 2, 2>;
  return per_sm == 1 ? (VrunKernel)k_vrun<MODEL, 1, 1> : (VrunKernel)k_vrun<MODEL, 1, 2>;
}

VrunKernel vrun_kernel(int model, int lanes, int per_sm) {
  switch (model) {
    case SPP_MODEL_VICSEK: return vrun_kernel_for<SPP_MODEL_VICSEK>(lanes, per_sm);
    case SPP_MODEL_VICSEK_REF_ANGLE: return vrun_kernel_for<SPP_MODEL_VICSEK_REF_ANGLE>(lanes, per_sm);
    case SPP_MODEL_VICSEK_REF_VECTOR: return vrun_kernel_for<SPP_MODEL_VICSEK_REF_VECTOR>(lanes, per_sm);
    default: return nullptr;
  }
}

}  // namespace

bool plan_vrun(const SppConsts& k, const DevState& d, VrunPlan* plan) {
  plan->blocks = 0;
  int dev = 0, sms = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop || sms < 1) {
    cudaGetLastError();
    return false;
  }
  /* As many lanes per particle as there is room for (us per step of the
   * vector rule, one GB300, lanes 1 / 2 / 4, before the walk without images: N =
   * 4,096 13.4 / 9.3 / 7.0; 43,776 18.1 / 13.6 / 13.2; 87,552 20.5 / 19.7); one block per SM while it holds
   * the threads. */
  const int64_t room = (int64_t)2 * sms * vrun_threads(2);
  const int lanes = 4 * (int64_t)d.n <= room ? 4 : (2 * (int64_t)d.n <= room ? 2 : 1);
  const int64_t total = (int64_t)d.n * lanes;
  if (total > room) return false;
  const int per_sm = total <= (int64_t)sms * vrun_threads(1) ? 1 : 2;
  /* The push past one block per SM is taken too, although its step kernels,
   * which have the registers, win in flocks: us per step resident / step
   * kernels 200 steps in at eta = 0.3, density 1 (2; 1/2): N = 97,001 55 / 57 (85 / 91;
   * 46 / 49), 100,001 65 / 61 (82 / 77; 52 / 50), 120,001 73 / 68 (114 / 102; 52 / 49),
   * 175,001 89 / 82 (108 / 97; 63 / 60).  From a uniform start it is the other way
   * round (upload, 10 steps, download: 120,001 370 / 446, with the first call's
   * graph capture 415 / 630; 175,001 412 / 533, 466 / 712).  The other rules stay
   * ahead in flocks as well (vector 27 / 31 at 175,001, angles 27 / 34). */
  int threads = (int)(((total + per_sm * sms - 1) / (per_sm * sms) + 31) / 32 * 32);
  if (threads < 128) threads = 128;
  const int blocks = (int)((total + threads - 1) / threads);
  VrunKernel f = vrun_kernel(k.model, lanes, per_sm);
  int fit = 0;
  if (!f || blocks > RUN_MAX_BLOCKS ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, f, threads, 0) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if ((int64_t)fit * sms < blocks) return false;
  plan->blocks = blocks;
  plan->threads = threads;
  plan->lanes = lanes;
  plan->per_sm = per_sm;
  const uint64_t cells = ((uint64_t)d.D * d.D + 3) & ~3ull;
  plan->cells = (uint32_t)cells;
  /* Bucket places per cell: 32, fewer (down to 4) where the cells are many for
   * the particles, so that a dilute system does not hold memory by its area:
   * at most 128 places per particle (density 1/4 with 32) or 2 million, and 12
   * million at all (32 bytes each, 40 with the angle rule's headings: 384 and
   * 480 MB); beyond that the general path (3,000 particles at L = 420 held 362
   * MB of buckets, 10 MB now).  A unit cell at the usual densities holds a few
   * particles; a step with a fuller cell goes through the sorted copy.  us per
   * step with 32 / 16 / 8 / 4 places and of the general path, flocked (eta =
   * 0.05, 3,000 steps on): N = 3,000 at density 0.1 5.0 / 5.0 / 10.8 / 11.1, 16.2;
   * 50,000 at 0.25, angles, 14.3 / 19.7 / 20.4 / 20.2, 29.4; 175,000 at 0.1 43.3
   * with any, 49.1. */
  const uint64_t most = std::min<uint64_t>(12u << 20, std::max<uint64_t>(128u * (uint64_t)d.n, 2u << 20));
  plan->cap = 32;
  while (plan->cap > 4 && cells * plan->cap > most) plan->cap /= 2;
  if (cells * plan->cap > most) plan->blocks = 0;
  return plan->blocks > 0;
}

int launch_vrun(const SppConsts& k, const DevState& d, const VrunPlan& plan, const VrunBufs& vb, int nsteps, int first,
                int every, unsigned long long* sums, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.gridDim = dim3(plan.blocks);
  cfg.blockDim = dim3(plan.threads);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, vrun_kernel(k.model, plan.lanes, plan.per_sm), k, d, vb, nsteps, first, every, sums) ==
                 cudaSuccess
             ? 0
             : -1;
}
