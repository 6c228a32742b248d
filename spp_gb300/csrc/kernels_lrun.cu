/*
 * kernels_lrun.cu -- resident Lyapunov runs: base and tangent dynamics and
 * their renormalisations in one cooperative launch, on sm_103a.
 *
 * k_lrun advances the continuous model and its K tangent vectors (the method
 * of kernels_lyap.cu, in place of LyapunovBox::Evolution_Reorthonormalize,
 * parallel/lyapunovbox.h:128-194) with every particle owned by LANES threads
 * for the whole launch: a thread holds the particle's state and its share of
 * the particle's tangent components in registers.  Base and tangent stage
 * walk the list once: a neighbour's state and the heading components of its
 * vectors are gathered together.  One grid barrier per stage; rebuilds as in
 * k_run.  The renormalisation runs in the same launch, with the arithmetic
 * and the summation trees of k_gram / k_chol / k_apply: every result is the
 * same bits as from the separate kernels.
 *
 * FP64 is the renormalisation's cost (this GPU issues about two FP64
 * operations per SM and cycle): the Gram matrix's fixed 64 blocks of 256
 * threads are dealt out in halves of its rows, so that 128 SMs work on it
 * instead of 64, and the factorisation runs in a warp (right-looking, one
 * entry per lane, each entry's subtractions in the order of
 * spp_cholesky_inverse) in every block redundantly, which saves a barrier.
 *
 * Measured (one GB300, N = 16,384, K = 8, RK4, renormalised every 10 steps; us
 * per step, step graphs -> this): uniform 85 -> 31, flocked (60% of the
 * particles in flocks, lists of up to 159) 113 -> 61.  The renormalisation is
 * about 5 us of a step; the rest is the chain of k_run's stages (barrier,
 * gathers of 48 bytes per neighbour, update) and, in flocks, the longest
 * segments.  Flocked, 3 / 4 / 6 neighbours in flight in long segments 68 / 71 /
 * 73 (2: 76), dealing the warps around the blocks 68 -> 61; at unit density
 * dealing costs 3%, so short lists keep consecutive slots.
 */
#include "spp_rebuild.cuh"
#include "spp_lyap.cuh"

namespace {

/* threads per block at most: 128 or 168 registers per thread */
__host__ __device__ constexpr int lrun_threads(int lanes) { return lanes == 1 ? 384 : 512; }

/* Rows of the packed Gram matrix in each of two halves of equal work. */
template <int KP>
__host__ __device__ constexpr int gram_half(int row) {
  return KP == 8 ? (row == 7 || row == 5 || row == 2 || row == 0 ? 0 : 1) : (row == 3 || row == 0 ? 0 : 1);
}

/* One half of the rows of block vb of k_gram: the same sums per virtual
 * thread, the same shuffles and the same order of warps. */
template <int KP, int HALF>
__device__ __forceinline__ void gram_task(const float* V, int len, int K, int vb, double* partial,
                                          double (*warp_part)[SPP_GRAM_ENTRIES]) {
  const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int stride = SPP_GRAM_BLOCKS * SPP_GRAM_THREADS;
  for (int w = threadIdx.x >> 5; w < SPP_GRAM_THREADS / 32; w += nwarps) {
    double g[KP * (KP + 1) / 2];
#pragma unroll
    for (int a = 0; a < KP; ++a)
#pragma unroll
      for (int b = 0; b <= a; ++b)
        if (gram_half<KP>(a) == HALF) g[a * (a + 1) / 2 + b] = 0.0;
    for (int e = vb * SPP_GRAM_THREADS + w * 32 + lane; e < len; e += stride) {
      double v[KP];
#pragma unroll
      for (int a = 0; a < KP; ++a) v[a] = a < K ? (double)V[(size_t)a * len + e] : 0.0;
#pragma unroll
      for (int a = 0; a < KP; ++a)
#pragma unroll
        for (int b = 0; b <= a; ++b)
          if (gram_half<KP>(a) == HALF) g[a * (a + 1) / 2 + b] = g[a * (a + 1) / 2 + b] + v[a] * v[b];
    }
#pragma unroll
    for (int a = 0; a < KP; ++a)
#pragma unroll
      for (int b = 0; b <= a; ++b)
        if (gram_half<KP>(a) == HALF && a < K) {
          double x = g[a * (a + 1) / 2 + b];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) x = x + __shfl_down_sync(0xffffffffu, x, o);
          if (lane == 0) warp_part[w][a * (a + 1) / 2 + b] = x;
        }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < K * (K + 1) / 2; q += blockDim.x) {
    int a = 0;
    while ((a + 1) * (a + 2) / 2 <= q) ++a;
    if (gram_half<KP>(a) != HALF) continue;
    double x = 0.0;
    for (int w = 0; w < SPP_GRAM_THREADS / 32; ++w) x = x + warp_part[w][q];
    partial[(size_t)vb * SPP_GRAM_ENTRIES + q] = x;
  }
  __syncthreads();
}

struct CholShared {
  double G[SPP_GRAM_ENTRIES];
  double R[SPP_LYAP_MAX][SPP_LYAP_MAX];
  double inv[SPP_LYAP_MAX], logr[SPP_LYAP_MAX];
  double rinv[SPP_LYAP_MAX * SPP_LYAP_MAX];
  int bad;
};

/* spp_cholesky_inverse (spp_physics.h) by the first warp of the block, every
 * entry's operations in its order. */
__device__ __forceinline__ void warp_cholesky(int K, CholShared* c) {
  const int lane = threadIdx.x & 31;
  bool bad = false;
  for (int j = 0; j < K; ++j) {
    const double d = c->G[spp_gram_index(j, j)];
    if (!(d > 0.0)) bad = true;
    const double rjj = sqrt(d), inv = 1.0 / rjj;
    if (lane == 0) {
      c->R[j][j] = rjj;
      c->inv[j] = inv;
    }
    if (lane > j && lane < K) c->R[j][lane] = c->G[spp_gram_index(lane, j)] * inv;
    __syncwarp();
    /* entries (a, b), a >= b > j, in turn */
    const int m = K - 1 - j;
    for (int e = lane; e < m * (m + 1) / 2; e += 32) {
      int a = 0;
      while ((a + 1) * (a + 2) / 2 <= e) ++a;
      const int b = e - a * (a + 1) / 2 + j + 1;
      a += j + 1;
      c->G[spp_gram_index(a, b)] -= c->R[j][b] * c->R[j][a];
    }
    __syncwarp();
  }
  if (lane < K) {
    c->logr[lane] = log(c->R[lane][lane]);
    c->rinv[lane * SPP_LYAP_MAX + lane] = c->inv[lane];
    for (int r = lane - 1; r >= 0; --r) {
      double v = 0.0;
      for (int q = r + 1; q <= lane; ++q) v += c->R[r][q] * c->rinv[q * SPP_LYAP_MAX + lane];
      c->rinv[r * SPP_LYAP_MAX + lane] = -v * c->inv[r];
    }
  }
  __syncwarp();
  if (bad)   /* dependent vectors: R^{-1} = 1 */
    for (int e = lane; e < SPP_LYAP_MAX * SPP_LYAP_MAX; e += 32) c->rinv[e] = e % (SPP_LYAP_MAX + 1) == 0;
  if (lane == 0) c->bad = bad;
}

/* The renormalisation of the vectors in L.t0 (two Cholesky-QR passes). */
template <int KP>
__device__ __noinline__ bool lrun_renormalize(const DevState& d, const LyapState& L, unsigned* target, unsigned* s_word,
                                              CholShared* c, double (*warp_part)[SPP_GRAM_ENTRIES]) {
  const int T = blockDim.x, tid = threadIdx.x, K = L.K, len = 3 * L.n;
  auto barrier = [&]() -> bool {
    *target += gridDim.x;
    __syncthreads();
    if (tid == 0) {
      grid_arrive(d.ctl);
      *s_word = grid_wait(d.ctl, *target);
    }
    __syncthreads();
    return *s_word != 0u;
  };
  for (int pass = 0; pass < 2; ++pass) {
    for (int task = blockIdx.x; task < 2 * SPP_GRAM_BLOCKS; task += gridDim.x) {
      if (task < SPP_GRAM_BLOCKS) gram_task<KP, 0>(L.t0, len, K, task, L.partial, warp_part);
      else gram_task<KP, 1>(L.t0, len, K, task - SPP_GRAM_BLOCKS, L.partial, warp_part);
    }
    if (!barrier()) return false;
    for (int q = tid; q < K * (K + 1) / 2; q += T) {
      double x = 0.0;
#pragma unroll 8
      for (int b = 0; b < SPP_GRAM_BLOCKS; ++b) x = x + L.partial[(size_t)b * SPP_GRAM_ENTRIES + q];
      c->G[q] = x;
    }
    __syncthreads();
    if (tid < 32) warp_cholesky(K, c);
    __syncthreads();
    if (blockIdx.x == 0 && tid < K) {
      if (c->bad) *L.error = 1u;
      else L.log_stretch[tid] = L.log_stretch[tid] + c->logr[tid];
    }
    for (int e = blockIdx.x * T + tid; e < len; e += gridDim.x * T) {
      double v[KP];
#pragma unroll
      for (int a = 0; a < KP; ++a) v[a] = a < K ? (double)L.t0[(size_t)a * len + e] : 0.0;
#pragma unroll
      for (int a = 0; a < KP; ++a) {
        if (a >= K) break;
        double x = 0.0;
#pragma unroll
        for (int b = 0; b <= a; ++b) x = x + v[b] * c->rinv[b * SPP_LYAP_MAX + a];
        L.t0[(size_t)a * len + e] = (float)x;
      }
    }
    if (!barrier()) return false;
  }
  return true;
}

/* nsteps steps, renormalised after the steps first, first + every, ... and,
 * with finish, after the last. */
template <int LANES, int KP>
__global__ void __launch_bounds__(lrun_threads(LANES), 1)
    k_lrun(const __grid_constant__ SppConsts k, const __grid_constant__ DevState d, const __grid_constant__ LyapState L,
           int nst, int nsteps, int first, int every, bool finish) {
  constexpr int VPL = KP / LANES;          /* vectors per lane: v = lane_r + LANES m */
  constexpr int GROUP = LANES == 1 ? 3 : 2;   /* neighbours gathered together */
  constexpr int BIG = 3;                      /* the same for long segments */
  extern __shared__ __align__(16) unsigned char lrun_smem[];
  __shared__ unsigned fin[2][2];
  __shared__ unsigned s_word;
  __shared__ CholShared chol;
  __shared__ double warp_part[SPP_GRAM_THREADS / 32][SPP_GRAM_ENTRIES];
  const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31;
  const int R = run_rows(d.cap, LANES, 1);
  int32_t* const rows = reinterpret_cast<int32_t*>(lrun_smem) + tid;                        /* [R][T] */
  unsigned long long* const keycol = reinterpret_cast<unsigned long long*>(lrun_smem) + tid; /* the rebuild's and the long sort's */
  Ctl* const ctl = d.ctl;
  const int n = d.n, K = L.K;
  /* Consecutive slots to consecutive threads; with long lists warp by warp
   * around the blocks, so that a flock's particles (neighbours in the slot
   * order) are spread over the SMs. */
  const int i = (R > RUN_ROWS ? ((tid >> 5) * (int)gridDim.x + (int)blockIdx.x) * 32 + lane : (int)blockIdx.x * T + tid) /
                LANES;
  const int lane_r = LANES == 1 ? 0 : tid % LANES;
  const bool inb = i < n;
  const bool head = inb && lane_r == 0;
  if (ctl->run_timeout) return;   /* the same for every block */
  uint32_t step = ctl->step;
  unsigned target = 0;
  auto barrier = [&]() -> bool {
    target += gridDim.x;
    __syncthreads();
    if (tid == 0) {
      grid_arrive(ctl);
      s_word = grid_wait(ctl, target);
    }
    __syncthreads();
    return s_word != 0u;
  };

  float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float th0 = 0.0f, dth = 0.0f;
  float2 rf = make_float2(0.0f, 0.0f);
  uint32_t pid = 0u;
  int q_begin = 0, len = 0;
  float t0[VPL][3], ta[VPL][3];   /* vectors at the start of the step, RK4 slope sums */
  float u[VPL];                   /* heading components of the stage input */
#pragma unroll
  for (int m = 0; m < VPL; ++m) {
    u[m] = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c) t0[m][c] = ta[m][c] = 0.0f;
  }
  const float* us = L.uslot;                                 /* [n][KP], this stage's */
  float* uo = L.uslot + (size_t)KP * (size_t)n;              /* the next stage's */
  bool wide = false;
  auto load_own = [&](bool with_list) {
    if (!inb) return;
    p = d.pos[i];
    pid = d.id[i];
    th0 = d.theta[i];
    rf = d.ref[i];
    if (!with_list) return;
    len = d.nn[i];
    if (LANES > 1) {
      const unsigned long long lc = d.nn_lanes[i];
      q_begin = 0;
      for (int r = 0; r < lane_r; ++r) q_begin += (int)((lc >> (16 * r)) & 0xffffull);
      len = (int)((lc >> (16 * lane_r)) & 0xffffull);
    }
    const int mr = len < R ? len : R;
    for (int q = 0; q < mr; q += 4) {
      int v[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) v[w] = q + w < mr ? d.nbr[(size_t)(q_begin + q + w) * n + i] : i;
#pragma unroll
      for (int w = 0; w < 4; ++w)
        if (q + w < mr) rows[(q + w) * T] = spp_index_ok(ctl, v[w], n) ? v[w] : i;
    }
  };
  auto load = [&](bool with_list) {
    load_own(with_list);
    wide = __reduce_max_sync(0xffffffffu, (unsigned)len) >= (unsigned)RUN_LONG;
  };
  /* the owner's vectors from and to L.t0 (by particle id) */
  auto fetch_vectors = [&]() {
    if (!inb) return;
#pragma unroll
    for (int m = 0; m < VPL; ++m) {
      const int v = lane_r + LANES * m;
      if (v < K)
#pragma unroll
        for (int c = 0; c < 3; ++c) t0[m][c] = L.t0[(size_t)(v * 3 + c) * n + pid];
    }
  };
  auto store_vectors = [&]() {
    if (!inb) return;
#pragma unroll
    for (int m = 0; m < VPL; ++m) {
      const int v = lane_r + LANES * m;
      if (v < K)
#pragma unroll
        for (int c = 0; c < 3; ++c) L.t0[(size_t)(v * 3 + c) * n + pid] = t0[m][c];
    }
  };
  /* the stage input's heading components to buf, in slot order */
  auto publish = [&](float* buf) {
    if (!inb) return;
#pragma unroll
    for (int m = 0; m < VPL; ++m) {
      const int v = lane_r + LANES * m;
      if (v < K) buf[(size_t)i * KP + v] = u[m];
    }
  };
  auto start_vectors = [&]() {
#pragma unroll
    for (int m = 0; m < VPL; ++m) u[m] = t0[m][2];
    publish(const_cast<float*>(us));
  };

  const int gthreads = gridDim.x * T, gtid = blockIdx.x * T + tid;
  for (uint32_t c = gtid; c < d.n_keys; c += gthreads) d.cell_count[c] = 0u;
  if (tid < 4) fin[tid >> 1][tid & 1] = 0u;
  bool frozen = ctl->frozen != 0u;   /* the same for every block: set by an earlier launch */
  load(!frozen);
  fetch_vectors();
  if (head) dth = spp_rot_noise(&k, pid, step);
  start_vectors();
  const float4* cur = d.pos;
  float4* oth = d.half;
  const float gp = k.g * k.one_minus_alpha_over_pi;
  if (!barrier()) return;

  int to_renorm = first;
  int t = 0;
  for (; t < nsteps && !frozen; ++t) {
    const float x0 = p.x, y0 = p.y;
    float kfx = 0.0f, kfy = 0.0f, ktq = 0.0f;
    unsigned decision = 1u;
    if (blockIdx.x == 0 && tid == 0) {
      ctl->run_disp[(t + 1) % 3] = 0u;
      ctl->run_step[(t + 1) % 3] = 0u;
    }
    for (int stage = 0; stage < nst; ++stage) {
      const bool last = stage == nst - 1;
      float disp2 = 0.0f, step2 = 0.0f;
      const int inner = !inb || (fabsf(p.x) < k.interior && fabsf(p.y) < k.interior);
      const int plain = __all_sync(0xffffffffu, inner);
      SppAccF a;
      spp_accf_zero(&a);
      float acc[KP];
      float4 ui[KP / 4];
#pragma unroll
      for (int g = 0; g < KP; ++g) acc[g] = 0.0f;
#pragma unroll
      for (int g = 0; g < KP / 4; ++g)
        ui[g] = inb ? reinterpret_cast<const float4*>(us + (size_t)i * KP)[g] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      /* one neighbour: the base stage's alignment sums and the vectors'
       * couplings */
      auto pair = [&](const float4& pj, const float4* uj) {
        float dx, dy;
        const float d2 = plain ? spp_pair_sep(&k, 0, p.x, p.y, pj.x, pj.y, &dx, &dy)
                               : spp_pair_sep(&k, 1, p.x, p.y, pj.x, pj.y, &dx, &dy);
        if (!(d2 < k.ral2)) return;
        const spp_f2 cs = spp_add2(spp_f2_make(a.sc, a.ss), spp_f2_make(pj.z, pj.w));
        a.sc = cs.x;
        a.ss = cs.y;
        const float cij = spp_tangent_coupling(p.z, p.w, pj.z, pj.w);
#pragma unroll
        for (int g = 0; g < KP / 4; ++g) {
          acc[4 * g] = acc[4 * g] + cij * (uj[g].x - ui[g].x);
          acc[4 * g + 1] = acc[4 * g + 1] + cij * (uj[g].y - ui[g].y);
          acc[4 * g + 2] = acc[4 * g + 2] + cij * (uj[g].z - ui[g].z);
          acc[4 * g + 3] = acc[4 * g + 3] + cij * (uj[g].w - ui[g].w);
        }
      };
      auto entry = [&](int q) -> int {
        const int j = q < R ? rows[q * T] : d.nbr[(size_t)(q_begin + q) * n + i];
        return spp_index_ok(ctl, j, n) ? j : i;
      };
      int q0 = 0;
      if (wide)
        for (; q0 + BIG <= len; q0 += BIG) {
          int jg[BIG];
          float4 pg[BIG], ug[BIG][KP / 4];
#pragma unroll
          for (int w = 0; w < BIG; ++w) jg[w] = entry(q0 + w);
#pragma unroll
          for (int w = 0; w < BIG; ++w) {
            pg[w] = cur[jg[w]];
#pragma unroll
            for (int g = 0; g < KP / 4; ++g) ug[w][g] = reinterpret_cast<const float4*>(us + (size_t)jg[w] * KP)[g];
          }
#pragma unroll
          for (int w = 0; w < BIG; ++w) pair(pg[w], ug[w]);
        }
      for (; q0 < len; q0 += GROUP) {
        int jg[GROUP];
        float4 pg[GROUP], ug[GROUP][KP / 4];
#pragma unroll
        for (int w = 0; w < GROUP; ++w) jg[w] = q0 + w < len ? entry(q0 + w) : i;
#pragma unroll
        for (int w = 0; w < GROUP; ++w) {
          pg[w] = cur[jg[w]];
#pragma unroll
          for (int g = 0; g < KP / 4; ++g) ug[w][g] = reinterpret_cast<const float4*>(us + (size_t)jg[w] * KP)[g];
        }
#pragma unroll
        for (int w = 0; w < GROUP; ++w)
          if (q0 + w < len) pair(pg[w], ug[w]);
      }
      /* lane sums as (p0 + p1) + (p2 + p3); each lane keeps its own vectors' */
      float mine[VPL];
      if (LANES == 4) {
        const bool odd = lane_r & 1, upper = lane_r & 2;
        float half[KP / 2];
#pragma unroll
        for (int m = 0; m < KP / 2; ++m) {
          const float keep = odd ? acc[2 * m + 1] : acc[2 * m], send = odd ? acc[2 * m] : acc[2 * m + 1];
          half[m] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
        }
#pragma unroll
        for (int m = 0; m < KP / 4; ++m) {
          const float keep = upper ? half[2 * m + 1] : half[2 * m], send = upper ? half[2 * m] : half[2 * m + 1];
          mine[m] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
          a.sc = a.sc + __shfl_xor_sync(0xffffffffu, a.sc, o);
          a.ss = a.ss + __shfl_xor_sync(0xffffffffu, a.ss, o);
        }
      } else {
#pragma unroll
        for (int m = 0; m < VPL; ++m) mine[m] = acc[m];
      }
      /* tangent stage */
#pragma unroll
      for (int m = 0; m < VPL; ++m) {
        const float slope[3] = {-k.v0 * p.w * u[m], k.v0 * p.z * u[m], gp * mine[m]};
        float un = 0.0f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float uc = 0.0f;
          if (stage == 0) ta[m][c] = 0.0f;
          spp_tangent_stage_update(&k, stage, nst, slope[c], &t0[m][c], &ta[m][c], &uc);
          if (c == 2) un = uc;
        }
        u[m] = last ? t0[m][2] : un;   /* the last stage's output is the next step's start */
      }
      publish(uo);
      /* base stage */
      if (head) {
        float fx, fy, tau;
        spp_abp_forces(&k, 0, &a, p.x, p.y, p.z, p.w, &fx, &fy, &tau);
        float h, frac;
        if (nst == 2) {
          h = stage == 0 ? k.half_dt : k.dt;
          frac = stage == 0 ? 0.5f : 1.0f;
        } else {
          if (stage == 0) {
            kfx = fx; kfy = fy; ktq = tau;
          } else if (stage < 3) {
            kfx = kfx + 2.0f * fx; kfy = kfy + 2.0f * fy; ktq = ktq + 2.0f * tau;
          } else {
            fx = kfx + fx; fy = kfy + fy; tau = ktq + tau;
          }
          h = stage < 2 ? k.half_dt : (stage == 2 ? k.dt : k.dt6);
          frac = stage < 2 ? 0.5f : 1.0f;
        }
        float nx, ny, nt, nc, ns;
        int gx = 0, gy = 0;
        spp_stage_update(h, frac, x0, y0, th0, fx, fy, tau, dth, &k, &nx, &ny, &nt, &nc, &ns, &gx, &gy, 0);
        p = make_float4(nx, ny, nc, ns);
        oth[i] = p;
        if (last) {
          th0 = nt;
          if (gx | gy) {
            const int2 g = d.img[i];
            d.img[i] = make_int2(g.x + gx, g.y + gy);
          }
          float ddx, ddy;
          disp2 = spp_sep_cl(&k, 0, nx, ny, rf.x, rf.y, &ddx, &ddy);
          step2 = spp_sep_cl(&k, 0, nx, ny, x0, y0, &ddx, &ddy);
        }
      }
      if (LANES > 1) {
        const int src = lane & ~(LANES - 1);
        p.x = __shfl_sync(0xffffffffu, p.x, src);
        p.y = __shfl_sync(0xffffffffu, p.y, src);
        p.z = __shfl_sync(0xffffffffu, p.z, src);
        p.w = __shfl_sync(0xffffffffu, p.w, src);
      }
      if (last) {
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
      if (last && head) dth = spp_rot_noise(&k, pid, step + 1u);
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
      float* const uwas = const_cast<float*>(us);
      us = uo;
      uo = uwas;
    }
    ++step;
    const bool rebuild = decision & 2u;
    const bool renorm = --to_renorm == 0 || (finish && t + 1 == nsteps);
    if (!rebuild && !renorm) continue;
    store_vectors();
    if (rebuild) {
      const int built = run_rebuild<LANES>(k, d, i, head, p, th0, pid, keycol, &target, &s_word);
      if (built == RUN_LOST) return;
      frozen = built == RUN_FROZEN;
      cur = d.pos;
      oth = d.half;
      load(!frozen);
      if (head) dth = spp_rot_noise(&k, pid, step);
      if (frozen) continue;   /* the renormalisations of the steps left out follow below */
    }
    if (renorm) {
      to_renorm = every;
      if (!barrier()) return;   /* every owner's vectors are in L.t0 */
      if (!lrun_renormalize<KP>(d, L, &target, &s_word, &chol, warp_part)) return;
    }
    fetch_vectors();
    start_vectors();
    if (!barrier()) return;
  }
  if (frozen) {
    /* a list overflowed: as in the step graphs, whose stages skip the steps
     * left but whose renormalisations run, from that of the last good step on;
     * the vectors are in L.t0 */
    if (!barrier()) return;
    const int done = t > 0 ? spp_events_upto(t - 1, first, every) : 0;
    const int all = spp_events_upto(nsteps, first, every) + (finish && spp_next_event(nsteps, first, every) != every);
    for (int c = done; c < all; ++c)
      if (!lrun_renormalize<KP>(d, L, &target, &s_word, &chol, warp_part)) return;
  } else {
    store_vectors();   /* those of a launch that ends between renormalisations */
  }

  if (head) {
    if (cur != d.pos) d.pos[i] = p;
    d.theta[i] = th0;
  }
  if (tid == 0) {
    if (blockIdx.x == 0) {
      ctl->step = step;
      ctl->need_rebuild = 0u;
    }
    /* the last block to leave clears the barrier for the next launch */
    __threadfence();
    if (atomicAdd(&ctl->run_exit, 1u) == gridDim.x - 1) {
      ctl->run_bar = 0u;
      ctl->run_exit = 0u;
      for (int c = 0; c < 3; ++c) ctl->run_disp[c] = ctl->run_step[c] = 0u;
    }
  }
}

typedef void (*LrunKernel)(SppConsts, DevState, LyapState, int, int, int, int, bool);

LrunKernel lrun_kernel(int lanes, int K) {
  if (lanes == SPP_GATHER_LANES) return K <= 4 ? (LrunKernel)k_lrun<4, 4> : (LrunKernel)k_lrun<4, 8>;
  return K <= 4 ? (LrunKernel)k_lrun<1, 4> : (LrunKernel)k_lrun<1, 8>;
}

}  // namespace

bool plan_lrun(const SppConsts& k, const DevState& d, int K, RunPlan* plan) {
  plan->blocks = 0;
  int dev = 0, sms = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop || sms < 1) {
    cudaGetLastError();
    return false;
  }
  const int lanes = k.lanes, most = lrun_threads(lanes);
  const int64_t total = (int64_t)d.n * lanes;
  if (total > (int64_t)sms * most) return false;
  int threads = (int)(((total + sms - 1) / sms + 31) / 32 * 32);
  if (threads < 128) threads = 128;
  const int blocks = (int)((total + threads - 1) / threads);
  LrunKernel f = lrun_kernel(lanes, K);
  int fit = 0;
  if (blocks > RUN_MAX_BLOCKS ||
      cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * RUN_ROWS_LONG * most) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, f, threads,
                                                    (size_t)4 * RUN_ROWS_LONG * threads) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if ((int64_t)fit * sms < blocks) return false;
  plan->blocks = blocks;
  plan->threads = threads;
  plan->per_sm = 1;
  return true;
}

int launch_lrun(const SppConsts& k, const DevState& d, const LyapState& L, const RunPlan& plan, int nstages, int nsteps,
                int first, int every, bool finish, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.gridDim = dim3(plan.blocks);
  cfg.blockDim = dim3(plan.threads);
  cfg.dynamicSmemBytes = (size_t)4 * run_rows(d.cap, k.lanes, 1) * plan.threads;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, lrun_kernel(k.lanes, L.K), k, d, L, nstages, nsteps, first, every, finish) ==
                 cudaSuccess
             ? 0
             : -1;
}
