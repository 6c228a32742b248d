/*
 * kernels_run.cu -- resident runs: many steps of a Verlet-list system in one
 * cooperative launch, on sm_103a.
 *
 * k_run advances nsteps whole steps (Box::Multi_Step, parallel/box.h:394-439)
 * with every particle owned by one thread (or by the k.lanes threads of its
 * neighbour sums) for the whole launch.  Per stage a thread gathers its
 * neighbours, writes its new stage state, and the grid meets at a barrier;
 * the list rebuild (count, scan, scatter, build) runs inside the same loop
 * when the step's displacements ask for it.  The arithmetic and its order
 * are those of k_abp_stage and of the rebuild kernels, so a run's bits do
 * not depend on which of the two advanced it.
 *
 * Why: below about 200,000 threads a stage launch is under one wave and is
 * bound by the latency of its dependent loads (list length -> list entry ->
 * neighbour state -> the particle's own inputs), the launch itself and the
 * end-of-step bookkeeping, 10 us per stage whatever the size.  Here the
 * particle's inputs stay in registers and its list in shared memory between
 * rebuilds, so a stage is one round of gathers plus one barrier.
 *
 * Measured on one GB300 (us per step, ABP at unit density; step graphs ->
 * resident): RK2 N = 16,384: 22 -> 8.6; RK2 N = 65,536: 23 -> 10.0; vesicles
 * (163,840 bodies, RK4): 38 -> 22.1.  A stage at N = 16,384 is about 6,300
 * cycles: 1,700 for the gathers and pair terms, 1,250 for the update, 1,700
 * until the block's stores are visible and its arrival is out, 1,500 to
 * 2,000 for the other blocks' arrivals.  What bounds it is that chain of L2
 * round trips, not a throughput; larger systems that do not fit stay with
 * the step graphs, whose stage launches are issue-bound (at N = 1M a
 * persistent grid was slower, 35.7 against 33.8 us per stage).
 */
#include "spp_internal.cuh"
#include "spp_rebuild.cuh"

namespace {

/* Threads per block at most, with one or two blocks per SM: 96 or 56
 * registers per thread. */
__host__ __device__ constexpr int run_threads(int per_sm) { return per_sm == 1 ? 640 : 576; }
constexpr int RING_SMEM = 16;            /* slots of the four ring neighbours (bead models) */
/* What a thread keeps of its particle between stages and does not need in
 * the neighbour walk: with one block per SM in registers, with two in shared
 * memory (as spilled local memory it would be refetched from L2 after every
 * barrier, whose acquire drops the SM's L1 lines). */
enum { C_X0, C_Y0, C_TH0, C_DTH, C_RFX, C_RFY, C_KFX, C_KFY, C_KTQ, C_WORDS };
constexpr int COLD_SMEM = C_WORDS * 4;   /* two blocks per SM */
template <int PER_SM>
struct Cold {
  float v[C_WORDS];
  __device__ __forceinline__ Cold(float*, int) {}
  __device__ __forceinline__ float& operator[](int q) { return v[q]; }
};
template <>
struct Cold<2> {
  float* col;
  int stride;
  __device__ __forceinline__ Cold(float* c, int s) : col(c), stride(s) {}
  __device__ __forceinline__ float& operator[](int q) { return col[q * stride]; }
};
/* Neighbour states gathered together.  Measured (us per RK2 / RK4 step, ABP
 * at unit density, groups of 2 / 4): one lane, one block per SM, N = 65,536:
 * 10.35 / 10.01 and 18.2 / 17.4; two blocks per SM (56 registers), N =
 * 163,840: 14.5 / 15.2 and 24.4 / 25.8; four lanes, N = 16,384: 8.6 / 8.7. */
/* Long segments (RUN_LONG) are walked 8 at a time instead: 16,384 particles of
 * the continuous model, 60% of them in flocks with lists of up to 159, 48 -> 41
 * us per RK4 step. */
__host__ __device__ constexpr int run_group(int lanes, int per_sm) { return lanes == 1 && per_sm == 1 ? 4 : 2; }

template <int LAW, int KIND>
__device__ __forceinline__ void run_pair(const SppConsts& k, const DevState& d, int wrap, SppAccF* a, int nbi, int j,
                                         float4 pi, float4 pj) {
  if (KIND == SPP_KIND_CHAIN) {
    const int nbj = d.id[j] < (uint32_t)k.n_beads ? 1 : k.chain_nb;
    spp_pair_chain(&k, LAW, wrap, a, nbi, nbj, pi.x, pi.y, pi.z, pi.w, pj.x, pj.y, pj.z, pj.w);
  } else {
    spp_pair_abp_lkwv(&k, LAW, KIND, wrap, a, pi.x, pi.y, pi.z, pi.w, pj.x, pj.y, pj.z, pj.w, 1);
  }
}

/* The system must hold a valid list (an upload or a completed step leaves
 * one).  Every block is resident (cooperative launch).  Two state buffers,
 * pos and half, alternate by stage: a stage reads one and writes the other,
 * and the barrier after it separates its reads from the next stage's writes.
 *
 * The step's largest displacements go through slot t % 3 of run_disp /
 * run_step: slot (t + 1) % 3 is cleared before the barrier of step t, after
 * every block has read it (that was before the barrier of step t - 1). */
template <int LAW, int KIND, int LANES, int CLOSED, int PER_SM>
__global__ void __launch_bounds__(run_threads(PER_SM), PER_SM) k_run(const __grid_constant__ SppConsts k, const __grid_constant__ DevState d,
                                                         int nst, int nsteps) {
  constexpr bool BEADLIKE = (KIND == SPP_KIND_BEADS || KIND == SPP_KIND_CHAIN);
  constexpr int GROUP = run_group(LANES, PER_SM);
  constexpr int BIG = PER_SM == 1 && KIND != SPP_KIND_CHAIN ? 8 : 0;   /* the same for long segments */
  extern __shared__ __align__(16) unsigned char run_smem[];
  __shared__ unsigned fin[2][2];
  __shared__ unsigned s_word;
  const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31;
  const int R = run_rows(d.cap, LANES, PER_SM);
  int32_t* const rows = reinterpret_cast<int32_t*>(run_smem) + tid;                        /* [R][T] */
  unsigned long long* const keycol = reinterpret_cast<unsigned long long*>(run_smem) + tid; /* the rebuild's and the long sort's */
  int32_t* const ring = reinterpret_cast<int32_t*>(run_smem + (size_t)R * 4 * T) + tid;     /* [4][T] */
  Cold<PER_SM> cold(reinterpret_cast<float*>(run_smem + (size_t)(R * 4 + (BEADLIKE ? RING_SMEM : 0)) * T) + tid, T);
  Ctl* const ctl = d.ctl;
  const int n = d.n;
  const int i = (blockIdx.x * T + tid) / LANES;
  const int lane_r = LANES == 1 ? 0 : tid % LANES;
  const bool inb = i < n;
  const bool head = inb && lane_r == 0;
  if (ctl->frozen || ctl->run_timeout) return;   /* the same for every block */
  uint32_t step = ctl->step;
  unsigned target = 0;

  float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  uint32_t pid = 0u;
  int q_begin = 0, len = 0;
  bool wide = false;
  /* the particle and its list from global memory (all threads call) */
  auto load_own = [&](bool with_list) {
    if (!inb) return;
    p = d.pos[i];
    pid = d.id[i];
    cold[C_TH0] = d.theta[i];
    const float2 rf = d.ref[i];
    cold[C_RFX] = rf.x;
    cold[C_RFY] = rf.y;
    if (!with_list) return;
    len = d.nn[i];
    if (LANES > 1) {
      const unsigned long long lc = d.nn_lanes[i];
      q_begin = 0;
      for (int r = 0; r < lane_r; ++r) q_begin += (int)((lc >> (16 * r)) & 0xffffull);
      len = (int)((lc >> (16 * lane_r)) & 0xffffull);
    }
    const int m = len < R ? len : R;
    for (int q = 0; q < m; q += 4) {
      int v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = q + u < m ? d.nbr[(size_t)(q_begin + q + u) * n + i] : i;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (q + u < m) rows[(q + u) * T] = spp_index_ok(ctl, v[u], n) ? v[u] : i;
    }
    if (BEADLIKE && pid < (uint32_t)k.n_beads) {
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        uint32_t slot = d.inv[spp_ring_neighbor(&k, pid, o < 2 ? o - 2 : o - 1)];
        if (!spp_index_ok(ctl, slot, n)) slot = (uint32_t)i;
        ring[o * T] = (int32_t)slot;
      }
    }
  };
  auto load = [&](bool with_list) {
    load_own(with_list);
    wide = __reduce_max_sync(0xffffffffu, (unsigned)len) >= (unsigned)RUN_LONG;
  };
  auto noise = [&](uint32_t at) -> float {
    if (!head || (BEADLIKE && pid < (uint32_t)k.n_beads)) return 0.0f;
    return spp_rot_noise(&k, pid, at);
  };

  const int gthreads = gridDim.x * T, gtid = blockIdx.x * T + tid;
  for (uint32_t c = gtid; c < d.n_keys; c += gthreads) d.cell_count[c] = 0u;
  if (tid < 4) fin[tid >> 1][tid & 1] = 0u;
  load(true);
  if (!(BEADLIKE && k.tumble)) cold[C_DTH] = noise(step);
  const float4* cur = d.pos;
  float4* oth = d.half;
  __syncthreads();

  for (int t = 0; t < nsteps; ++t) {
    cold[C_X0] = p.x;
    cold[C_Y0] = p.y;
    unsigned decision = 1u;
    if (BEADLIKE && k.tumble)
      cold[C_DTH] = head && pid >= (uint32_t)k.n_beads ? spp_tumble_noise(&k, pid, step, d.tumble + pid) : 0.0f;
    if (blockIdx.x == 0 && tid == 0) {
      ctl->run_disp[(t + 1) % 3] = 0u;
      ctl->run_step[(t + 1) % 3] = 0u;
    }
    for (int stage = 0; stage < nst; ++stage) {
      const bool last = stage == nst - 1;
      float disp2 = 0.0f, step2 = 0.0f;
      SppAccF a;
      spp_accf_zero(&a);
      const int nbi = (KIND == SPP_KIND_CHAIN && pid >= (uint32_t)k.n_beads) ? k.chain_nb : 1;
      const int inner = !inb || (fabsf(p.x) < k.interior && fabsf(p.y) < k.interior);
      const int plain = CLOSED || __all_sync(0xffffffffu, inner);
      float4 rp[4];
      const int bead = BEADLIKE && head && pid < (uint32_t)k.n_beads;
      if (BEADLIKE && bead) {
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          const float2 v = reinterpret_cast<const float2*>(cur)[2 * (size_t)ring[o * T]];
          rp[o] = make_float4(v.x, v.y, 0.0f, 0.0f);
        }
      }
      int q0 = 0;
      if (BIG > 0 && wide)
        for (; q0 + BIG <= len; q0 += BIG) {
          int jg[BIG > 0 ? BIG : 1];
          float4 pg[BIG > 0 ? BIG : 1];
#pragma unroll
          for (int u = 0; u < BIG; ++u) {
            const int q = q0 + u;
            jg[u] = q < R ? rows[q * T] : d.nbr[(size_t)(q_begin + q) * n + i];
            if (!spp_index_ok(ctl, jg[u], n)) jg[u] = i;
          }
#pragma unroll
          for (int u = 0; u < BIG; ++u) pg[u] = cur[jg[u]];
#pragma unroll
          for (int u = 0; u < BIG; ++u) {
            if (plain) run_pair<LAW, KIND>(k, d, 0, &a, nbi, jg[u], p, pg[u]);
            else run_pair<LAW, KIND>(k, d, 1, &a, nbi, jg[u], p, pg[u]);
          }
        }
      for (; q0 < len; q0 += GROUP) {
        int jg[GROUP];
        float4 pg[GROUP];
#pragma unroll
        for (int u = 0; u < GROUP; ++u) {
          const int q = q0 + u;
          jg[u] = q < len ? (q < R ? rows[q * T] : d.nbr[(size_t)(q_begin + q) * n + i]) : i;
          if (!spp_index_ok(ctl, jg[u], n)) jg[u] = i;
        }
#pragma unroll
        for (int u = 0; u < GROUP; ++u) pg[u] = cur[jg[u]];
#pragma unroll
        for (int u = 0; u < GROUP; ++u)
          if (q0 + u < len) {
            if (plain) run_pair<LAW, KIND>(k, d, 0, &a, nbi, jg[u], p, pg[u]);
            else run_pair<LAW, KIND>(k, d, 1, &a, nbi, jg[u], p, pg[u]);
          }
      }
      if (LANES > 1) {
#pragma unroll
        for (int o = 1; o < LANES; o <<= 1) {
          a.fx = a.fx + __shfl_xor_sync(0xffffffffu, a.fx, o);
          a.fy = a.fy + __shfl_xor_sync(0xffffffffu, a.fy, o);
          a.ss = a.ss + __shfl_xor_sync(0xffffffffu, a.ss, o);
          a.sc = a.sc + __shfl_xor_sync(0xffffffffu, a.sc, o);
          a.tq = a.tq + __shfl_xor_sync(0xffffffffu, a.tq, o);
          a.cnt += __shfl_xor_sync(0xffffffffu, a.cnt, o);
          a.ovf |= __shfl_xor_sync(0xffffffffu, a.ovf, o);
        }
      }
      if (head) {
        if (LAW == SPP_FORCE_R12_TRUNC && a.ovf) atomicOr(&ctl->fx_overflow, 1u);
        const float x0 = cold[C_X0], y0 = cold[C_Y0], th0 = cold[C_TH0], dth = cold[C_DTH];
        float fx, fy, tau;
        if (BEADLIKE) {
          float rfx = 0.0f, rfy = 0.0f;
          if (bead) {
            const float px[5] = {rp[0].x, rp[1].x, p.x, rp[2].x, rp[3].x};
            const float py[5] = {rp[0].y, rp[1].y, p.y, rp[2].y, rp[3].y};
            spp_ring_forces(&k, px, py, &rfx, &rfy);
          }
          if (KIND == SPP_KIND_CHAIN && !bead) spp_chain_velocity(&k, &a, p.z, p.w, p.z, p.w, &fx, &fy, &tau);
          else spp_bead_velocity(&k, !bead, &a, rfx, rfy, p.z, p.w, &fx, &fy, &tau);
        } else {
          spp_abp_forces(&k, CLOSED, &a, p.x, p.y, p.z, p.w, &fx, &fy, &tau);
        }
        if (KIND == SPP_KIND_CHAIN && !bead && nst == 1) {
          /* Move() turns first and projects the force on the new heading */
          float wc, ws;
          spp_sincosf(spp_euler_theta(&k, th0, tau, dth), &ws, &wc);
          spp_chain_velocity(&k, &a, p.z, p.w, wc, ws, &fx, &fy, &tau);
        }
        float nx, ny, nt, nc, ns;
        int gx = 0, gy = 0;
        if (nst == 1) {
          spp_euler_update(x0, y0, th0, fx, fy, tau, dth, &k, &nx, &ny, &nt, &nc, &ns, &gx, &gy, CLOSED);
        } else {
          float h, frac;
          if (nst == 2) {
            h = stage == 0 ? k.half_dt : k.dt;
            frac = stage == 0 ? 0.5f : 1.0f;
          } else {
            if (stage == 0) {
              cold[C_KFX] = fx; cold[C_KFY] = fy; cold[C_KTQ] = tau;
            } else if (stage < 3) {
              cold[C_KFX] = cold[C_KFX] + 2.0f * fx;
              cold[C_KFY] = cold[C_KFY] + 2.0f * fy;
              cold[C_KTQ] = cold[C_KTQ] + 2.0f * tau;
            } else {
              fx = cold[C_KFX] + fx; fy = cold[C_KFY] + fy; tau = cold[C_KTQ] + tau;
            }
            h = stage < 2 ? k.half_dt : (stage == 2 ? k.dt : k.dt6);
            frac = stage < 2 ? 0.5f : 1.0f;
          }
          spp_stage_update(h, frac, x0, y0, th0, fx, fy, tau, dth, &k, &nx, &ny, &nt, &nc, &ns, &gx, &gy, CLOSED);
        }
        p = make_float4(nx, ny, nc, ns);
        oth[i] = p;
        if (last) {
          cold[C_TH0] = nt;
          if (gx | gy) {
            const int2 g = d.img[i];
            d.img[i] = make_int2(g.x + gx, g.y + gy);
          }
          float ddx, ddy;
          disp2 = spp_sep_cl(&k, CLOSED, nx, ny, cold[C_RFX], cold[C_RFY], &ddx, &ddy);
          step2 = spp_sep_cl(&k, CLOSED, nx, ny, x0, y0, &ddx, &ddy);
        }
      }
      if (LANES > 1) {
        p.x = __shfl_sync(0xffffffffu, p.x, lane & ~(LANES - 1));
        p.y = __shfl_sync(0xffffffffu, p.y, lane & ~(LANES - 1));
        p.z = __shfl_sync(0xffffffffu, p.z, lane & ~(LANES - 1));
        p.w = __shfl_sync(0xffffffffu, p.w, lane & ~(LANES - 1));
      }
      if (last) {
        /* the block's largest displacements: float bits of non-negative
         * values, so the unsigned maximum is the float maximum */
        const unsigned m1 = __reduce_max_sync(0xffffffffu, __float_as_uint(disp2));
        const unsigned m2 = __reduce_max_sync(0xffffffffu, __float_as_uint(step2));
        if (lane == 0) {
          atomicMax(&fin[t & 1][0], m1);
          atomicMax(&fin[t & 1][1], m2);
        }
      }
      target += gridDim.x;
      __syncthreads();
      if (tid == 0) {
        if (last) {
          if (fin[t & 1][0]) atomicMax(&ctl->run_disp[t % 3], fin[t & 1][0]);
          if (fin[t & 1][1]) atomicMax(&ctl->run_step[t % 3], fin[t & 1][1]);
          fin[t & 1][0] = 0u;
          fin[t & 1][1] = 0u;
        }
        grid_arrive(ctl);
      }
      /* the next step's noise while the other blocks arrive */
      if (last && !(BEADLIKE && k.tumble)) cold[C_DTH] = noise(step + 1u);
      if (tid == 0) {
        unsigned w = grid_wait(ctl, target) ? 1u : 0u;
        if (w && last) {
          /* the rebuild rule of finish_step (kernels_step.cu) */
          const unsigned b1 = ld_relaxed(&ctl->run_disp[t % 3]), b2 = ld_relaxed(&ctl->run_step[t % 3]);
          const float dm = sqrtf(__uint_as_float(b1)), sm = sqrtf(__uint_as_float(b2));
          if (k.half_skin > 0.0f) {
            if (dm + 2.0f * sm > k.half_skin) w |= 2u;
            if (blockIdx.x == 0 && dm > k.half_skin) atomicAdd(&ctl->late_rebuilds, 1u);
          }
        }
        s_word = w;
      }
      __syncthreads();
      decision = s_word;
      if (!(decision & 1u)) return;
      float4* const was = const_cast<float4*>(cur);
      cur = oth;
      oth = was;
    }
    ++step;
    if (!(decision & 2u)) continue;

    const int built = run_rebuild<LANES>(k, d, i, head, p, cold[C_TH0], pid, keycol, &target, &s_word);
    if (built == RUN_LOST) return;
    cur = d.pos;
    oth = d.half;
    load(built == RUN_BUILT);
    if (built == RUN_FROZEN) break;
    if (!(BEADLIKE && k.tumble)) cold[C_DTH] = noise(step);
  }

  if (head) {
    if (cur != d.pos) d.pos[i] = p;
    d.theta[i] = cold[C_TH0];
  }
  if (tid == 0) {
    if (blockIdx.x == 0) {
      ctl->step = step;
      ctl->need_rebuild = 0u;
    }
    /* the last block to leave clears the barrier for the next launch: by
     * then every block has passed its last wait */
    __threadfence();
    if (atomicAdd(&ctl->run_exit, 1u) == gridDim.x - 1) {
      ctl->run_bar = 0u;
      ctl->run_exit = 0u;
      for (int c = 0; c < 3; ++c) ctl->run_disp[c] = ctl->run_step[c] = 0u;
    }
  }
}

typedef void (*RunKernel)(SppConsts, DevState, int, int);

template <int PER_SM>
RunKernel run_kernel_for(const SppConsts& k, int lanes) {
  const int kind = spp_pair_kind(&k);
  const bool four = lanes == SPP_GATHER_LANES;
#define SPP_RUN_CASE(L, K)                                                                                    \
  if (k.force_law == L && kind == K)                                                                          \
    return four ? (RunKernel)k_run<L, K, SPP_GATHER_LANES, 0, PER_SM> : (RunKernel)k_run<L, K, 1, 0, PER_SM>;
#define SPP_RUN_CASE_W(L, K)                                                                                  \
  if (k.force_law == L && kind == K && k.closed)                                                              \
    return four ? (RunKernel)k_run<L, K, SPP_GATHER_LANES, 1, PER_SM> : (RunKernel)k_run<L, K, 1, 1, PER_SM>; \
  SPP_RUN_CASE(L, K)
  SPP_RUN_CASE_W(SPP_FORCE_HARMONIC, SPP_KIND_ABP)
  SPP_RUN_CASE_W(SPP_FORCE_R12_TRUNC, SPP_KIND_ABP)
  SPP_RUN_CASE_W(SPP_FORCE_NONE, SPP_KIND_ABP)
  SPP_RUN_CASE_W(SPP_FORCE_NONE, SPP_KIND_CONT)
  SPP_RUN_CASE_W(SPP_FORCE_NONE, SPP_KIND_CONT_ALPHA)
  SPP_RUN_CASE(SPP_FORCE_R12_TRUNC, SPP_KIND_BEADS)
  SPP_RUN_CASE(SPP_FORCE_HARMONIC, SPP_KIND_BEADS)
  SPP_RUN_CASE(SPP_FORCE_NONE, SPP_KIND_BEADS)
#undef SPP_RUN_CASE
#undef SPP_RUN_CASE_W
  if (kind == SPP_KIND_CHAIN && k.force_law == SPP_FORCE_R12_TRUNC)
    return (RunKernel)k_run<SPP_FORCE_R12_TRUNC, SPP_KIND_CHAIN, 1, 0, PER_SM>;
  if (kind == SPP_KIND_CHAIN && k.force_law == SPP_FORCE_NONE)
    return (RunKernel)k_run<SPP_FORCE_NONE, SPP_KIND_CHAIN, 1, 0, PER_SM>;
  return nullptr;
}

RunKernel run_kernel(const SppConsts& k, int lanes, int per_sm) {
  return per_sm == 1 ? run_kernel_for<1>(k, lanes) : run_kernel_for<2>(k, lanes);
}

int run_lanes(const SppConsts& k) { return spp_pair_kind(&k) == SPP_KIND_CHAIN ? 1 : k.lanes; }

size_t run_smem_bytes(const SppConsts& k, int rows, int per_sm, int threads) {
  return (size_t)(4 * rows + (k.model == SPP_MODEL_BEADS ? RING_SMEM : 0) + (per_sm == 2 ? COLD_SMEM : 0)) * threads;
}

}  // namespace

bool plan_run(const SppConsts& k, const DevState& d, RunPlan* plan) {
  plan->blocks = plan->threads = 0;
  const int lanes = run_lanes(k);
  int dev = 0, sms = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop || sms < 1) {
    cudaGetLastError();
    return false;
  }
  /* one block per SM while a block holds its share of the threads, else two */
  const int64_t total = (int64_t)d.n * lanes;
  const int per_sm = total <= (int64_t)sms * run_threads(1) ? 1 : 2;
  if (total > (int64_t)per_sm * sms * run_threads(per_sm)) return false;
  int threads = (int)(((total + per_sm * sms - 1) / (per_sm * sms) + 31) / 32 * 32);
  if (threads < 128) threads = 128;
  const int blocks = (int)((total + threads - 1) / threads);
  RunKernel f = run_kernel(k, lanes, per_sm);
  if (!f || blocks > RUN_MAX_BLOCKS) return false;
  const int most = per_sm == 1 ? RUN_ROWS_LONG : RUN_ROWS;   /* the list may grow */
  int fit = 0;
  if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)run_smem_bytes(k, most, per_sm, run_threads(per_sm))) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, f, threads, run_smem_bytes(k, most, per_sm, threads)) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if ((int64_t)fit * sms < blocks) return false;
  plan->blocks = blocks;
  plan->threads = threads;
  plan->per_sm = per_sm;
  return true;
}

int launch_run(const SppConsts& k, const DevState& d, const RunPlan& plan, int nstages, int nsteps, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.gridDim = dim3(plan.blocks);
  cfg.blockDim = dim3(plan.threads);
  cfg.dynamicSmemBytes = run_smem_bytes(k, run_rows(d.cap, run_lanes(k), plan.per_sm), plan.per_sm, plan.threads);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, run_kernel(k, run_lanes(k), plan.per_sm), k, d, nstages, nsteps) == cudaSuccess ? 0 : -1;
}
