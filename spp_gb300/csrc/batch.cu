/*
 * batch.cu -- many independent Vicsek systems in one set of launches.
 *
 * The reference runs a parameter sweep as a task farm: serial/mpi-main.cpp:
 * 157-176 hands noise values round-robin to MPI ranks, each rank running
 * whole independent boxes one after another.  Here every system of the
 * sweep lives in one set of device arrays, indexed by a per-system offset
 * table (particle range, cell range, constants, activity, step count), and
 * each phase of a step is ONE launch over all particles of all systems:
 *   scan of the cell counts (two launches) | k_batch_scatter | k_batch_step |
 *   k_batch_finish
 * k_batch_step also counts the particles into the cells of the next step, so
 * k_batch_bin runs only when the state or the set of active systems is new.
 * Small systems (1k particles) that alone could not fill the GPU share it
 * with the large ones; the step loop is captured in CUDA graphs.  Retired or
 * finished systems stay in place and are copied through without work.
 *
 * Per-system observables are accumulated on the device every step: the
 * polarization P = |sum (cos, sin)| / N (exact fixed-point sums), its first
 * four moments over a start-up window, and its mean over a stationary
 * window -- the inputs and targets of the sweep surrogate.
 */
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <string>
#include <vector>
#include "spp_internal.cuh"
#include "spp_batch.cuh"
#include "spp_pack.cuh"

namespace {

/* Compact particle index t -> (system, slot). */
__device__ __forceinline__ int act_slot(const DevBatch& b, int t, int* s) {
  *s = (int)b.act_sys[t];
  return t + b.sact[*s].a_corr;
}

/* Counts particle t, at (x, y), into the compact cells of the next step: its
 * cell (cx | cy << 16) and its place in it.  Keys are compact cell indices: a
 * system's D x D row-major grid starts at its a_coff, so the scan runs over
 * the cells of active systems only and a system's cell starts, plus its
 * a_corr, are slots of its own particle range. */
__device__ __forceinline__ void count_particle(const DevBatch& b, const BatchSys& S, uint32_t a_coff, int t, float x,
                                               float y) {
  const int cx = spp_cell_coord(x, S.k.L, S.k.L2, (int)S.D, SPP_BIN_GEOMETRIC);
  const int cy = spp_cell_coord(y, S.k.L, S.k.L2, (int)S.D, SPP_BIN_GEOMETRIC);
  const uint32_t key = a_coff + (uint32_t)cy * S.D + (uint32_t)cx;
  b.cell[t] = (uint32_t)cx | (uint32_t)cy << 16;
  b.rank[t] = atomicAdd(&b.cell_count[key], 1u);   /* moved particles rarely share a cell with their warp */
}

__global__ void __launch_bounds__(SPP_BLOCK) k_batch_bin(DevBatch b) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= b.n_act) return;
  int s;
  const int i = act_slot(b, t, &s);
  const float2 p = *reinterpret_cast<const float2*>(b.ent + i);
  count_particle(b, b.sys[s], b.sact[s].a_coff, t, p.x, p.y);
}

/* Into cell order, within each system's range.  A system that has finished
 * since the compact space was built stays in place.  THETA: the rules that
 * read headings (all but the vector sum, whose step needs none). */
template <bool THETA>
__global__ void __launch_bounds__(SPP_BLOCK) k_batch_scatter(DevBatch b) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= b.n_act) return;
  int s;
  const int i = act_slot(b, t, &s);
  const uint32_t cell = b.cell[t];
  const SysAct A = b.sact[s];
  const BatchSys& S = b.sys[s];
  const uint32_t key = A.a_coff + (cell >> 16) * S.D + (cell & 0xffffu);
  const uint32_t dst = S.active ? b.cell_start[key] + b.rank[t] + (uint32_t)A.a_corr : (uint32_t)i;
  b.ent_alt[dst] = b.ent[i];
  b.id_alt[dst] = b.id[i];
  b.cell_alt[dst] = cell;
  if (THETA) b.theta_alt[dst] = b.theta[i];
}

/* Models of the batch step kernel: one rule for all systems of the batch
 * (the common case), or any mix (runtime dispatch per system). */
constexpr int BATCH_MIXED = -1;

/* The sums a particle receives. */
struct BatchAcc {
  PackedSum cx, cy;       /* headings of the aligning neighbours */
  SppAcc a;               /* count, angles (ax, ay: the push terms) */
};

/* One candidate (entry q, heading thj for the angle rule) at separation
 * (dx, dy), self: the particle itself. */
template <int MODEL>
__device__ __forceinline__ void visit(const SppConsts& k, float dx, float dy, float4 q, const float* thj, bool self,
                                      BatchAcc* acc) {
  const int model = MODEL == BATCH_MIXED ? k.model : MODEL;
  const float d2 = fmaf(dx, dx, dy * dy);
  if (!(d2 < k.ral2)) return;
  if (model != SPP_MODEL_VICSEK && self) return;   /* the vector sum counts the particle itself */
  acc->a.cnt += 1;
  if (model == SPP_MODEL_VICSEK_REF_ANGLE) {
    spp_fx_add_guarded(&acc->a.at, *thj, &acc->a.ovf);
    return;
  }
  packed_add(&acc->cx, q.z);
  packed_add(&acc->cy, q.w);
  if (model == SPP_MODEL_VICSEK_REF_VECTOR && d2 < k.rpush2 && d2 > 0.0f) spp_push_vicsek(&k, &acc->a, dx, dy, d2);
}

/* Walks the n cell-ordered slots from lo on, UNROLL at a time with their
 * loads first.  (sx, sy): what the minimum image subtracts from every
 * separation of these cells. */
template <int MODEL, int UNROLL>
__device__ __forceinline__ void walk(const DevBatch& b, const SppConsts& k, float2 p, float sx, float sy, int i,
                                     uint32_t lo, int n, BatchAcc* acc) {
  const float4* e = b.ent_alt + lo;
  for (int t = 0; t < n; t += UNROLL, e += UNROLL) {
    float4 q[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      if (t + u < n) q[u] = __ldg(e + u);
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      if (t + u < n) {
        const spp_f2 r = spp_sub2(spp_sub2(spp_f2_make(p.x, p.y), spp_f2_make(q[u].x, q[u].y)), spp_f2_make(sx, sy));
        const uint32_t j = lo + (uint32_t)(t + u);
        visit<MODEL>(k, r.x, r.y, q[u], b.theta_alt + j, (int)j == i, acc);
      }
  }
}

/* The slots of the columns ca .. cb of the three rows around cell (., cy) and
 * the rows' image shifts. */
__device__ __forceinline__ void segments(const DevBatch& b, const BatchSys* S, SysAct A, int cy, int ca, int cb,
                                         uint32_t (&lo)[3], int (&len)[3]) {
  const int D = (int)S->D;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    int ny = cy + r - 1;
    ny = ny < 0 ? ny + D : (ny >= D ? ny - D : ny);
    const uint32_t row = A.a_coff + (uint32_t)ny * (uint32_t)D;
    const uint32_t first = b.cell_start[row + (uint32_t)ca];
    lo[r] = first + (uint32_t)A.a_corr;
    len[r] = (int)(b.cell_start[row + (uint32_t)cb + 1u] - first);   /* one start past the last cell */
  }
}

/* One Vicsek step of every active system (VicsekParticle{,2}::Interact/Move,
 * shared/particle.h:145-247, or the arg-sum rule), from the cell-ordered
 * copy back into the primary arrays; per-system heading sums for P.
 *
 * Candidates: the 3x3 cells around a particle are, per grid row, one run of
 * consecutive keys (row-major keys), i.e. one contiguous range of the
 * cell-ordered arrays, walked one row after the other; the column that the
 * periodic wrap adds (a particle in the first or last column) is three more
 * ranges.  The minimum image needs no comparison: what it subtracts is the
 * same number for every candidate of a range, 0 or +-2 L (where the two
 * differ, which takes a candidate two cells or more away, both separations
 * are beyond every cutoff, so neither is used).
 *
 * Measured, full 512-point sweep (7.4M particles, us per batched step over the
 * first 32 steps / after 300): 771 / 1,126 at first.  One 16-byte entry per
 * candidate instead of 24 bytes, 56 instead of 92 bytes per particle moved by
 * the scatter (headings and box crossings no longer travel), the binning pass
 * folded in here (20 bytes read again, a launch), a two-launch scan that
 * clears the counts (25 us instead of 90: k_scan_counts) and the bookkeeping
 * beside the scan: 504 / 822.  Row by row instead of the three rows flattened
 * into one sequence with comparisons for the image (about 20 instructions a
 * candidate -> 13): 479 / 674; systems ordered by expected flocks: 471 / 561.
 * What bounds it: issue (77% of the slots), the
 * walk's loads, and lanes that wait for their warp's longest rows (22 of 32
 * active).
 * Slower: blocks of 64 or 128 threads (less L1 reuse, 634 and 616 against 605
 * some 200 steps in), a second copy of the walk without the image shift (811:
 * spills), the rows as a rolled loop (617). */
template <int MODEL, int UNROLL, int MIN_BLOCKS>
__global__ void __launch_bounds__(SPP_BLOCK, MIN_BLOCKS) k_batch_step(DevBatch b) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  int hx = 0, lx = 0, hy = 0, ly = 0;
  int s = -1, i = -1;
  int active = 0;
  const BatchSys* S = nullptr;
  SysAct A = {0u, 0};
  float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  BatchAcc acc;
  acc.cx = acc.cy = {0, 0};
  spp_acc_zero(&acc.a);
  if (t < b.n_act) {
    i = act_slot(b, t, &s);
    S = &b.sys[s];
    A = b.sact[s];
    active = (int)S->active;
    p = b.ent_alt[i];
  }
  if (active) {
    const SppConsts& k = S->k;
    const int D = (int)S->D;
    const uint32_t cell = b.cell_alt[i];
    const int cx = (int)(cell & 0xffffu), cy = (int)(cell >> 16);
    const float L2 = k.L2;
    uint32_t lo[3];
    int len[3];
    segments(b, S, A, cy, max(cx - 1, 0), min(cx + 1, D - 1), lo, len);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const float sy = r == 0 && cy == 0 ? -L2 : (r == 2 && cy == D - 1 ? L2 : 0.0f);
      walk<MODEL, UNROLL>(b, k, make_float2(p.x, p.y), 0.0f, sy, i, lo[r], len[r], &acc);
    }
    if (cx == 0 || cx == D - 1) {   /* the column that the periodic wrap adds */
      const int cw = cx == 0 ? D - 1 : 0;
      segments(b, S, A, cy, cw, cw, lo, len);
#pragma unroll 1
      for (int r = 0; r < 3; ++r) {
        const float sy = r == 0 && cy == 0 ? -L2 : (r == 2 && cy == D - 1 ? L2 : 0.0f);
        const uint32_t l = r == 0 ? lo[0] : (r == 1 ? lo[1] : lo[2]);
        const int n = r == 0 ? len[0] : (r == 1 ? len[1] : len[2]);
        walk<MODEL, UNROLL < 2 ? UNROLL : 2>(b, k, make_float2(p.x, p.y), cx == 0 ? -L2 : L2, sy, i, l, n, &acc);
      }
    }
  }
  if (active) {
    const SppConsts& k = S->k;
    if (acc.a.ovf) atomicOr(&b.ctl->fx_overflow, 1u);
    const spp_fx fx = packed_value(acc.cx, acc.a.cnt), fy = packed_value(acc.cy, acc.a.cnt);
    if (MODEL != SPP_MODEL_VICSEK_REF_ANGLE) {   /* (a mixed batch's angle rule does not read them) */
      acc.a.ax.hi += fx.hi;
      acc.a.ax.lo += fx.lo;
      acc.a.ay.hi += fy.hi;
      acc.a.ay.lo += fy.lo;
    }
    const uint32_t id = b.id_alt[i];
    float th0 = 0.0f, c0 = 0.0f, s0 = 0.0f;
    if (MODEL != SPP_MODEL_VICSEK) {
      th0 = b.theta_alt[i];
      spp_sincosf(th0, &s0, &c0);   /* as the step before left them */
    }
    const spp_u32x4 r = spp_draw(k.seed, k.system, id, S->steps, SPP_RNG_VICSEK);
    float x, y, c, sn, th;
    int gx = 0, gy = 0;
    spp_vicsek_update(&k, &acc.a, p.x, p.y, th0, c0, s0, r.v[0], &x, &y, &th, &c, &sn, &gx, &gy);
    const spp_fx px = fx_parts(c), py = fx_parts(sn);
    hx = px.hi; lx = px.lo; hy = py.hi; ly = py.lo;
    p = make_float4(x, y, pack_parts(px), pack_parts(py));
    b.ent[i] = p;
    b.theta[i] = th;
    b.id[i] = id;
    if (gx | gy) {   /* box crossings, by particle */
      int2* const g = b.img + S->p_off + id;
      *g = make_int2(g->x + gx, g->y + gy);
    }
  }
  if (i >= 0) count_particle(b, *S, A.a_coff, t, p.x, p.y);
  if (!active) s = -1;  /* no contribution */
  /* heading sums: one atomic per group of lanes of the same system (|hi| <=
   * 32 and |lo| <= 2^21, so 32 of them fit a word) */
  const unsigned peers = __all_sync(0xffffffffu, s == __shfl_sync(0xffffffffu, s, 0)) ? 0xffffffffu
                                                                                     : __match_any_sync(0xffffffffu, s);
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(peers) - 1;
  const int shx = __reduce_add_sync(peers, hx), slx = __reduce_add_sync(peers, lx);
  const int shy = __reduce_add_sync(peers, hy), sly = __reduce_add_sync(peers, ly);
  if (lane == leader && s >= 0) {
    const spp_fx sx = {shx, slx}, sy = {shy, sly};
    atomicAdd(reinterpret_cast<unsigned long long*>(&b.stats[s].sx), (unsigned long long)spp_fx_units(sx));
    atomicAdd(reinterpret_cast<unsigned long long*>(&b.stats[s].sy), (unsigned long long)spp_fx_units(sy));
  }
}

/* Per system: P of the step just taken, moment sums, step counter, and the
 * stop at max_steps. */
__global__ void k_batch_finish(DevBatch b) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= b.n_sys) return;
  BatchSys& S = b.sys[s];
  BatchStats& T = b.stats[s];
  if (!S.active) return;
  const double inv = 7.450580596923828125e-09;  /* 2^-27 */
  const double px = (double)T.sx * inv / S.n, py = (double)T.sy * inv / S.n;
  const double P = sqrt(px * px + py * py);
  T.sx = 0;
  T.sy = 0;
  const uint32_t t = S.steps + 1u;  /* steps completed after this one */
  if ((int)t <= b.window) {
    const double P2 = P * P;
    T.w1 += P;
    T.w2 += P2;
    T.w3 += P2 * P;
    T.w4 += P2 * P2;
  }
  if ((int)t > b.stationary_from) {
    T.s1 += P;
    T.s2 += P * P;
    T.s4 += (P * P) * (P * P);
    T.ns += 1;
  }
  T.p_last = P;
  S.steps = t;
  if (b.max_steps > 0 && (int)t >= b.max_steps) S.active = 0u;
}

__global__ void k_batch_flags(DevBatch b) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < b.n_sys) b.flags[s] = b.sys[s].active;
}

/* The smallest uploaded particle with a non-finite value and the smallest
 * outside its system's box, into Ctl::bad_*. */
__global__ void k_batch_check(DevBatch b, const float* __restrict__ x, const float* __restrict__ y,
                              const float* __restrict__ th) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.n_total) return;
  const float xi = x[i], yi = y[i], L = b.sys[b.sys_of[i]].k.L;
  if (!isfinite(xi) || !isfinite(yi) || !isfinite(th[i])) atomicMin(&b.ctl->bad_nonfinite, (uint32_t)i);
  else if (xi < -L || xi >= L || yi < -L || yi >= L) atomicMin(&b.ctl->bad_range, (uint32_t)i);
}

__global__ void k_batch_init(DevBatch b, const float* x, const float* y, const float* th) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.n_total) return;
  float s, c;
  spp_sincosf(th[i], &s, &c);
  b.ent[i] = make_float4(x[i], y[i], pack_parts(fx_parts(c)), pack_parts(fx_parts(s)));
  b.theta[i] = th[i];
  b.img[i] = make_int2(0, 0);
  b.id[i] = (uint32_t)i - b.sys[b.sys_of[i]].p_off;
}

__global__ void k_batch_gather(DevBatch b, float* x, float* y, float* th, int32_t* img_x, int32_t* img_y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.n_total) return;
  const BatchSys& S = b.sys[b.sys_of[i]];
  const uint32_t dst = S.p_off + b.id[i];
  const float2 p = *reinterpret_cast<const float2*>(b.ent + i);
  x[dst] = p.x;
  y[dst] = p.y;
  th[dst] = b.theta[i];
  const int2 g = b.img[i];   /* by particle already */
  img_x[i] = g.x;
  img_y[i] = g.y;
}

__global__ void k_batch_set_active(DevBatch b, const int32_t* idx, int count, uint32_t value) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < count) {
    const int s = idx[q];
    if (s >= 0 && s < b.n_sys) {
      /* a system that reached max_steps stays finished */
      const int finished = b.max_steps > 0 && (int)b.sys[s].steps >= b.max_steps;
      b.sys[s].active = (value && !finished) ? 1u : 0u;
    }
  }
}

int bfail(int status, const std::string& m) {
  spp_internal_set_error(m.c_str());
  return status;
}

#define BCUDA(expr)                                                                     \
  do {                                                                                  \
    cudaError_t _e = (expr);                                                            \
    if (_e != cudaSuccess) return bfail(SPP_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(_e)); \
  } while (0)

inline int nblocks(int n) { return (n + SPP_BLOCK - 1) / SPP_BLOCK; }

}  // namespace

struct SppBatch {
  DevBatch d;
  std::vector<BatchSys> host_sys;
  uint32_t n_keys = 0;
  cudaStream_t stream = nullptr;
  cudaStream_t side = nullptr;      /* the forked branch of a captured step */
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  float *stage_x = nullptr, *stage_y = nullptr, *stage_t = nullptr;
  int32_t *stage_ix = nullptr, *stage_iy = nullptr;
  std::vector<std::pair<int, cudaGraphExec_t>> graphs;
  std::vector<cudaGraph_t> graph_defs;
  int64_t launches = 0;
  bool uploaded = false;
  int model = -1;  /* the one model of all systems, or -1 for a mix */
  std::vector<uint32_t> act_flags;  /* the active set the compact launch space was built for */
  bool act_valid = false;
  bool counted = false;             /* cell_count, cell and rank are those of the current state */
};

namespace {

template <class T>
int balloc(T** p, size_t count) {
  *p = nullptr;
  cudaError_t e = cudaMalloc((void**)p, (count ? count : 1) * sizeof(T));
  if (e != cudaSuccess) {
    *p = nullptr;
    return bfail(SPP_ERR_ALLOC, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  }
  return SPP_OK;
}

void batch_free(SppBatch* b) {
  for (auto& g : b->graphs) cudaGraphExecDestroy(g.second);
  for (auto g : b->graph_defs) cudaGraphDestroy(g);
  b->graphs.clear();
  b->graph_defs.clear();
  DevBatch& d = b->d;
  void* ptrs[] = {d.sys, d.stats, d.sys_of, d.ent, d.ent_alt, d.theta, d.theta_alt, d.img, d.id, d.id_alt,
                  d.cell, d.cell_alt, d.rank, d.cell_count, d.cell_start, d.scan_tmp, d.ctl, d.act_sys, d.sact,
                  d.flags, b->stage_x, b->stage_y, b->stage_t, b->stage_ix, b->stage_iy};
  for (void* q : ptrs)
    if (q) cudaFree(q);
  memset(&b->d, 0, sizeof(b->d));
  if (b->stream) cudaStreamDestroy(b->stream);
  if (b->side) cudaStreamDestroy(b->side);
  if (b->ev_fork) cudaEventDestroy(b->ev_fork);
  if (b->ev_join) cudaEventDestroy(b->ev_join);
  b->stream = b->side = nullptr;
  b->ev_fork = b->ev_join = nullptr;
}

/* Shapes of the step kernel <rule, candidates in flight, blocks per SM>.
 * Measured on one GB300 (us per batched step over the first 32 steps / after
 * 300, flocking):
 *   vector sum   <., 4, 5>        <., 2, 8>
 *     834k       60 / 128         57 / 143
 *     1.8M       138 / 176        130 / 192
 *     3.6M       268 / 330        241 / 293
 *     7.4M       540 / 650        479 / 567
 * Small batches wait on their longest walks, large ones want the warps.
 * Angles: <., 2, 8> 63 / 66 and 525 / 552 (834k, 7.4M); <., 4, 5>, measured
 * with the systems in the caller's order, 69 / 75 against 68 / 77 and 576 /
 * 613 against 525 / 550.  The push needs registers: <., 1, 5> 90 / 432 and 811 /
 * 1548, <., 2, 5> 95 / 464 and 853 / 1654, <., 4, 4> 96 / 407 and 897 / 1698;
 * mixed batches the same order (82 / 205 and 720 / 1116, 92 / 241 and 796 /
 * 1275, 92 / 198 and 839 / 1283). */
constexpr int BATCH_LARGE = 2500000;

/* One step, captured on st.  The per-system bookkeeping (k_batch_finish) runs
 * beside the next step's scan: it forks off after the step kernel and is
 * joined before the scatter, the first to read its results (`forked`: a
 * branch of the step before is open). */
int enqueue_batch_step(SppBatch* b, cudaStream_t st, bool forked) {
  const DevBatch& d = b->d;
  const int nb = nblocks(d.n_act);
  launch_scan_counts(d.cell_count, (uint32_t)d.n_act_keys, d.scan_tmp, d.cell_start, st);
  if (forked) BCUDA(cudaStreamWaitEvent(st, b->ev_join, 0));
  if (b->model == SPP_MODEL_VICSEK) k_batch_scatter<false><<<nb, SPP_BLOCK, 0, st>>>(d);
  else k_batch_scatter<true><<<nb, SPP_BLOCK, 0, st>>>(d);
  switch (b->model) {
    case SPP_MODEL_VICSEK:
      if (d.n_act >= BATCH_LARGE) k_batch_step<SPP_MODEL_VICSEK, 2, 8><<<nb, SPP_BLOCK, 0, st>>>(d);
      else k_batch_step<SPP_MODEL_VICSEK, 4, 5><<<nb, SPP_BLOCK, 0, st>>>(d);
      break;
    case SPP_MODEL_VICSEK_REF_ANGLE: k_batch_step<SPP_MODEL_VICSEK_REF_ANGLE, 2, 8><<<nb, SPP_BLOCK, 0, st>>>(d); break;
    case SPP_MODEL_VICSEK_REF_VECTOR: k_batch_step<SPP_MODEL_VICSEK_REF_VECTOR, 1, 5><<<nb, SPP_BLOCK, 0, st>>>(d); break;
    default: k_batch_step<BATCH_MIXED, 1, 5><<<nb, SPP_BLOCK, 0, st>>>(d); break;
  }
  BCUDA(cudaEventRecord(b->ev_fork, st));
  BCUDA(cudaStreamWaitEvent(b->side, b->ev_fork, 0));
  k_batch_finish<<<(d.n_sys + 31) / 32, 32, 0, b->side>>>(d);
  BCUDA(cudaEventRecord(b->ev_join, b->side));
  BCUDA(cudaGetLastError());
  return SPP_OK;
}

constexpr int BATCH_GRAPH_CHUNK = 32;

void batch_drop_graphs(SppBatch* b) {
  for (auto& g : b->graphs) cudaGraphExecDestroy(g.second);
  for (auto g : b->graph_defs) cudaGraphDestroy(g);
  b->graphs.clear();
  b->graph_defs.clear();
}

/* Reads the active flags and, when the set of active systems changed since
 * the compact launch space was built, rebuilds it (and the step graphs,
 * whose launch sizes depend on it). */
int batch_refresh_active(SppBatch* b) {
  DevBatch& d = b->d;
  const int ns = d.n_sys;
  k_batch_flags<<<nblocks(ns), SPP_BLOCK, 0, b->stream>>>(d);
  b->launches += 1;
  std::vector<uint32_t> flags((size_t)ns);
  BCUDA(cudaMemcpyAsync(flags.data(), d.flags, sizeof(uint32_t) * ns, cudaMemcpyDeviceToHost, b->stream));
  BCUDA(cudaStreamSynchronize(b->stream));
  if (b->act_valid && flags == b->act_flags) return SPP_OK;
  std::vector<SysAct> sact((size_t)ns);
  std::vector<uint32_t> act_sys;
  act_sys.reserve((size_t)d.n_total);
  uint32_t a_poff = 0, a_coff = 0;
  /* Where flocks are to be expected first: their walks are the longest, and
   * started last they would leave the GPU waiting for them.  Density over
   * noise (noise alone comes close, density alone does not); us per step over the
   * steps 300 to 332, in the caller's order / this: 64 points 149 / 128, 256
   * points 348 / 292, 512 points 671 / 562; unflocked 68 / 60, 246 / 239, 483 /
   * 472.  By size, largest first: 148, 357, 724. */
  auto flocks = [&](int s) {
    const BatchSys& S = b->host_sys[(size_t)s];
    const float w = (float)S.n / ((float)S.D * (float)S.D * (S.k.eta + 0.01f));
    return std::isfinite(w) ? w : 0.0f;
  };
  std::vector<int> order((size_t)ns);
  for (int s = 0; s < ns; ++s) order[(size_t)s] = s;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return flocks(x) > flocks(y); });
  for (int s : order) {
    const BatchSys& S = b->host_sys[(size_t)s];
    sact[(size_t)s] = {0u, 0};
    if (!flags[(size_t)s]) continue;
    sact[(size_t)s] = {a_coff, (int32_t)S.p_off - (int32_t)a_poff};
    act_sys.insert(act_sys.end(), S.n, (uint32_t)s);
    a_poff += S.n;
    a_coff += S.D * S.D;
  }
  BCUDA(cudaMemcpyAsync(d.sact, sact.data(), sizeof(SysAct) * ns, cudaMemcpyHostToDevice, b->stream));
  if (a_poff)
    BCUDA(cudaMemcpyAsync(d.act_sys, act_sys.data(), sizeof(uint32_t) * a_poff, cudaMemcpyHostToDevice,
                          b->stream));
  BCUDA(cudaStreamSynchronize(b->stream));
  batch_drop_graphs(b);
  d.n_act = (int)a_poff;
  d.n_act_keys = (int)a_coff;
  b->act_flags = flags;
  b->act_valid = true;
  b->counted = false;
  return SPP_OK;
}

int batch_graph(SppBatch* b, int nsteps, cudaGraphExec_t* out) {
  for (auto& g : b->graphs)
    if (g.first == nsteps) { *out = g.second; return SPP_OK; }
  cudaGraph_t graph = nullptr;
  BCUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
  int rc = SPP_OK;
  for (int i = 0; i < nsteps && rc == SPP_OK; ++i) rc = enqueue_batch_step(b, b->stream, i > 0);
  if (rc == SPP_OK && nsteps > 0 && cudaStreamWaitEvent(b->stream, b->ev_join, 0) != cudaSuccess)
    rc = bfail(SPP_ERR_CUDA, "capture: join");
  cudaError_t e = cudaStreamEndCapture(b->stream, &graph);
  if (rc != SPP_OK) { if (graph) cudaGraphDestroy(graph); return rc; }
  if (e != cudaSuccess) return bfail(SPP_ERR_CUDA, std::string("capture: ") + cudaGetErrorString(e));
  cudaGraphExec_t exec;
  e = cudaGraphInstantiate(&exec, graph, 0);
  if (e != cudaSuccess) {
    cudaGraphDestroy(graph);
    return bfail(SPP_ERR_CUDA, std::string("instantiate: ") + cudaGetErrorString(e));
  }
  b->graphs.push_back({nsteps, exec});
  b->graph_defs.push_back(graph);
  *out = exec;
  return SPP_OK;
}

int batch_step_enqueue(SppBatch* b, int nsteps) {
  if (b->d.n_act == 0) return SPP_OK;  /* nothing active */
  if (nsteps > 0 && !b->counted) {
    BCUDA(cudaMemsetAsync(b->d.cell_count, 0, sizeof(uint32_t) * (size_t)b->d.n_act_keys, b->stream));
    k_batch_bin<<<nblocks(b->d.n_act), SPP_BLOCK, 0, b->stream>>>(b->d);
    BCUDA(cudaGetLastError());
    b->launches += 1;
    b->counted = true;
  }
  while (nsteps > 0) {
    int chunk = nsteps >= BATCH_GRAPH_CHUNK ? BATCH_GRAPH_CHUNK : nsteps;
    cudaGraphExec_t exec;
    int rc = batch_graph(b, chunk, &exec);
    if (rc != SPP_OK) return rc;
    BCUDA(cudaGraphLaunch(exec, b->stream));
    b->launches += (int64_t)chunk * 5;
    nsteps -= chunk;
  }
  return SPP_OK;
}


}  // namespace

extern "C" {

int spp_batch_create(const SppParams* systems, int n_systems, SppBatch** out) {
  if (!systems || !out || n_systems < 1) return bfail(SPP_ERR_INVALID, "bad arguments");
  *out = nullptr;
  SppBatch* b = new SppBatch();
  b->host_sys.resize((size_t)n_systems);
  uint64_t p_off = 0, c_off = 0;
  for (int s = 0; s < n_systems; ++s) {
    const SppParams& p = systems[s];
    if (p.struct_size != sizeof(SppParams) || p.n < 1 || !(p.L > 0) || !(p.r_align > 0) ||
        (p.model != SPP_MODEL_VICSEK && p.model != SPP_MODEL_VICSEK_REF_ANGLE &&
         p.model != SPP_MODEL_VICSEK_REF_VECTOR) || p.boundary != SPP_BOUNDARY_PERIODIC) {
      delete b;
      return bfail(SPP_ERR_INVALID, "system " + std::to_string(s) +
                                        ": batches hold periodic Vicsek-family systems with n >= 1, L > 0");
    }
    double rc = p.r_align;
    if (p.model == SPP_MODEL_VICSEK_REF_VECTOR && p.r_push > rc) rc = p.r_push;
    int D = (int)std::floor(2.0 * p.L / (rc * 1.001));
    if (D < 3) {
      delete b;
      return bfail(SPP_ERR_INVALID, "system " + std::to_string(s) + ": box too small (2L/r < 3)");
    }
    b->model = s == 0 ? p.model : (b->model == p.model ? b->model : -1);
    BatchSys& S = b->host_sys[(size_t)s];
    memset(&S, 0, sizeof(S));
    spp_consts_from_params(&S.k, &p);
    S.p_off = (uint32_t)p_off;
    S.n = (uint32_t)p.n;
    S.c_off = (uint32_t)c_off;
    S.D = (uint32_t)D;
    S.active = 1u;
    S.steps = 0u;
    p_off += (uint64_t)p.n;
    c_off += (uint64_t)D * (uint64_t)D;
  }
  if (p_off > 0x7fffffffULL || c_off > scan_max_elements()) {
    delete b;
    return bfail(SPP_ERR_INVALID, "batch too large (particles or cells)");
  }
  DevBatch& d = b->d;
  memset(&d, 0, sizeof(d));
  d.n_total = (int)p_off;
  d.n_sys = n_systems;
  b->n_keys = (uint32_t)c_off;
  d.window = 500;
  d.stationary_from = 0;
  d.max_steps = 0;
  size_t n = (size_t)p_off;
  int rc = SPP_OK;
  rc = rc ? rc : balloc(&d.sys, (size_t)n_systems);
  rc = rc ? rc : balloc(&d.stats, (size_t)n_systems);
  rc = rc ? rc : balloc(&d.sys_of, n);
  rc = rc ? rc : balloc(&d.ent, n);
  rc = rc ? rc : balloc(&d.ent_alt, n);
  rc = rc ? rc : balloc(&d.theta, n);
  rc = rc ? rc : balloc(&d.theta_alt, b->model == SPP_MODEL_VICSEK ? 1 : n);
  rc = rc ? rc : balloc(&d.img, n);
  rc = rc ? rc : balloc(&d.id, n);
  rc = rc ? rc : balloc(&d.id_alt, n);
  rc = rc ? rc : balloc(&d.cell, n);
  rc = rc ? rc : balloc(&d.cell_alt, n);
  rc = rc ? rc : balloc(&d.rank, n);
  rc = rc ? rc : balloc(&d.cell_count, (size_t)c_off);
  rc = rc ? rc : balloc(&d.cell_start, (size_t)c_off + 1);
  rc = rc ? rc : balloc(&d.scan_tmp, ((size_t)c_off + 4095) / 4096 + 1);
  rc = rc ? rc : balloc(&d.ctl, 1);
  rc = rc ? rc : balloc(&d.act_sys, n);
  rc = rc ? rc : balloc(&d.sact, (size_t)n_systems);
  rc = rc ? rc : balloc(&d.flags, (size_t)n_systems);
  rc = rc ? rc : balloc(&b->stage_x, n);
  rc = rc ? rc : balloc(&b->stage_y, n);
  rc = rc ? rc : balloc(&b->stage_t, n);
  rc = rc ? rc : balloc(&b->stage_ix, n);
  rc = rc ? rc : balloc(&b->stage_iy, n);
  if (rc != SPP_OK) {
    batch_free(b);
    delete b;
    return rc;
  }
  std::vector<uint32_t> sys_of(n);
  for (int s = 0; s < n_systems; ++s)
    for (uint32_t q = 0; q < b->host_sys[s].n; ++q) sys_of[b->host_sys[s].p_off + q] = (uint32_t)s;
  cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->side, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_fork, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_join, cudaEventDisableTiming);
  /* on the batch's own stream, which does not wait for the legacy one */
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d.sys, b->host_sys.data(), sizeof(BatchSys) * n_systems, cudaMemcpyHostToDevice, b->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d.sys_of, sys_of.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice, b->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d.stats, 0, sizeof(BatchStats) * n_systems, b->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d.ctl, 0, sizeof(Ctl), b->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);   /* sys_of goes out of scope */
  if (e != cudaSuccess) {
    batch_free(b);
    delete b;
    return bfail(SPP_ERR_CUDA, std::string("batch setup: ") + cudaGetErrorString(e));
  }
  *out = b;
  return SPP_OK;
}

int spp_batch_destroy(SppBatch* b) {
  if (!b) return SPP_OK;
  if (b->stream) cudaStreamSynchronize(b->stream);
  batch_free(b);
  delete b;
  return SPP_OK;
}

int spp_batch_set_windows(SppBatch* b, int window_steps, int stationary_from, int max_steps) {
  if (!b || window_steps < 0 || stationary_from < 0 || max_steps < 0)
    return bfail(SPP_ERR_INVALID, "bad arguments");
  BCUDA(cudaStreamSynchronize(b->stream));
  for (auto& g : b->graphs) cudaGraphExecDestroy(g.second);
  for (auto g : b->graph_defs) cudaGraphDestroy(g);
  b->graphs.clear();
  b->graph_defs.clear();
  b->d.window = window_steps;
  b->d.stationary_from = stationary_from;
  b->d.max_steps = max_steps;
  return SPP_OK;
}

int spp_batch_upload(SppBatch* b, const float* x, const float* y, const float* theta, int total_n) {
  if (!b || !x || !y || !theta) return bfail(SPP_ERR_INVALID, "NULL argument");
  if (total_n != b->d.n_total) return bfail(SPP_ERR_INVALID, "total_n differs from the batch size");
  const size_t bytes = sizeof(float) * (size_t)total_n;
  BCUDA(cudaMemcpyAsync(b->stage_x, x, bytes, cudaMemcpyHostToDevice, b->stream));
  BCUDA(cudaMemcpyAsync(b->stage_y, y, bytes, cudaMemcpyHostToDevice, b->stream));
  BCUDA(cudaMemcpyAsync(b->stage_t, theta, bytes, cudaMemcpyHostToDevice, b->stream));
  /* checked on the device, before anything of the batch's state changes (the
   * host took 2 ms per million particles) */
  uint32_t bad[2] = {0xffffffffu, 0xffffffffu};
  static_assert(offsetof(Ctl, bad_range) == offsetof(Ctl, bad_nonfinite) + sizeof(uint32_t), "read together");
  BCUDA(cudaMemcpyAsync(&b->d.ctl->bad_nonfinite, bad, sizeof(bad), cudaMemcpyHostToDevice, b->stream));
  k_batch_check<<<nblocks(total_n), SPP_BLOCK, 0, b->stream>>>(b->d, b->stage_x, b->stage_y, b->stage_t);
  b->launches += 1;
  BCUDA(cudaMemcpyAsync(bad, &b->d.ctl->bad_nonfinite, sizeof(bad), cudaMemcpyDeviceToHost, b->stream));
  BCUDA(cudaStreamSynchronize(b->stream));
  if (bad[0] < bad[1]) return bfail(SPP_ERR_NUMERIC, "non-finite input at particle " + std::to_string(bad[0]));
  if (bad[1] != 0xffffffffu)
    return bfail(SPP_ERR_INVALID, "position outside its system's box at particle " + std::to_string(bad[1]));
  /* reset per-system counters and statistics */
  for (auto& S : b->host_sys) { S.active = 1u; S.steps = 0u; }
  BCUDA(cudaMemcpyAsync(b->d.sys, b->host_sys.data(), sizeof(BatchSys) * b->host_sys.size(),
                        cudaMemcpyHostToDevice, b->stream));
  BCUDA(cudaMemsetAsync(b->d.stats, 0, sizeof(BatchStats) * b->host_sys.size(), b->stream));
  k_batch_init<<<nblocks(b->d.n_total), SPP_BLOCK, 0, b->stream>>>(b->d, b->stage_x, b->stage_y,
                                                                      b->stage_t);
  b->launches += 1;
  BCUDA(cudaStreamSynchronize(b->stream));
  b->uploaded = true;
  b->counted = false;
  return SPP_OK;
}

int spp_batch_step(SppBatch* b, int nsteps) {
  if (!b || nsteps < 0) return bfail(SPP_ERR_INVALID, "bad arguments");
  if (!b->uploaded) return bfail(SPP_ERR_INVALID, "no state uploaded");
  int rc = batch_refresh_active(b);
  if (rc != SPP_OK) return rc;
  return batch_step_enqueue(b, nsteps);
}

int spp_batch_poll(SppBatch* b, SppSweepStats* out, int n_systems) {
  if (!b || !out || n_systems != b->d.n_sys) return bfail(SPP_ERR_INVALID, "bad arguments");
  BCUDA(cudaStreamSynchronize(b->stream));
  std::vector<BatchSys> sys((size_t)n_systems);
  std::vector<BatchStats> st((size_t)n_systems);
  Ctl c;
  BCUDA(cudaMemcpy(sys.data(), b->d.sys, sizeof(BatchSys) * n_systems, cudaMemcpyDeviceToHost));
  BCUDA(cudaMemcpy(st.data(), b->d.stats, sizeof(BatchStats) * n_systems, cudaMemcpyDeviceToHost));
  BCUDA(cudaMemcpy(&c, b->d.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost));
  if (c.fx_overflow) return bfail(SPP_ERR_OVERFLOW, "fixed-point range exceeded");
  for (int s = 0; s < n_systems; ++s) {
    SppSweepStats& o = out[s];
    memset(&o, 0, sizeof(o));
    const BatchStats& T = st[(size_t)s];
    const int64_t nw = (int64_t)(sys[s].steps < (uint32_t)b->d.window ? sys[s].steps : (uint32_t)b->d.window);
    o.steps = sys[s].steps;
    o.active = (int32_t)sys[s].active;
    o.p_last = T.p_last;
    o.window_steps = nw;
    if (nw > 0) {
      const double m1 = T.w1 / nw, m2 = T.w2 / nw, m3 = T.w3 / nw, m4 = T.w4 / nw;
      const double var = m2 - m1 * m1;
      o.p_mean = m1;
      o.p_var = var;
      const double c4 = m4 - 4 * m3 * m1 + 6 * m2 * m1 * m1 - 3 * m1 * m1 * m1 * m1;
      o.p_kurt = var > 0 ? c4 / (var * var) : 0.0;
    }
    o.stationary_steps = T.ns;
    if (T.ns > 0) {
      o.p_stationary = T.s1 / T.ns;
      o.p2_stationary = T.s2 / T.ns;
      o.p4_stationary = T.s4 / T.ns;
      if (o.p2_stationary > 0) {
        o.binder = 1.0 - o.p4_stationary / (3.0 * o.p2_stationary * o.p2_stationary);
        o.binder_reference = 1.0 - o.p4_stationary / (3.0 * o.p2_stationary);
      }
    }
  }
  return SPP_OK;
}

static int batch_set_active(SppBatch* b, const int32_t* systems, int count, uint32_t value) {
  if (!b || (count > 0 && !systems) || count < 0) return bfail(SPP_ERR_INVALID, "bad arguments");
  if (count == 0) return SPP_OK;
  int32_t* d_idx = nullptr;
  int rc = balloc(&d_idx, (size_t)count);
  if (rc != SPP_OK) return rc;
  BCUDA(cudaMemcpyAsync(d_idx, systems, sizeof(int32_t) * count, cudaMemcpyHostToDevice, b->stream));
  k_batch_set_active<<<nblocks(count), SPP_BLOCK, 0, b->stream>>>(b->d, d_idx, count, value);
  b->launches += 1;
  cudaError_t e = cudaStreamSynchronize(b->stream);
  cudaFree(d_idx);
  if (e != cudaSuccess) return bfail(SPP_ERR_CUDA, cudaGetErrorString(e));
  return SPP_OK;
}

int spp_batch_retire(SppBatch* b, const int32_t* systems, int count) {
  return batch_set_active(b, systems, count, 0u);
}

int spp_batch_resume(SppBatch* b, const int32_t* systems, int count) {
  return batch_set_active(b, systems, count, 1u);
}

int spp_batch_download(SppBatch* b, float* x, float* y, float* theta, int32_t* img_x,
                       int32_t* img_y, int total_n) {
  if (!b || !x || !y || !theta || total_n != b->d.n_total) return bfail(SPP_ERR_INVALID, "bad arguments");
  k_batch_gather<<<nblocks(total_n), SPP_BLOCK, 0, b->stream>>>(b->d, b->stage_x, b->stage_y,
                                                                  b->stage_t, b->stage_ix, b->stage_iy);
  b->launches += 1;
  size_t bytes = sizeof(float) * (size_t)total_n;
  BCUDA(cudaMemcpyAsync(x, b->stage_x, bytes, cudaMemcpyDeviceToHost, b->stream));
  BCUDA(cudaMemcpyAsync(y, b->stage_y, bytes, cudaMemcpyDeviceToHost, b->stream));
  BCUDA(cudaMemcpyAsync(theta, b->stage_t, bytes, cudaMemcpyDeviceToHost, b->stream));
  if (img_x) BCUDA(cudaMemcpyAsync(img_x, b->stage_ix, bytes, cudaMemcpyDeviceToHost, b->stream));
  if (img_y) BCUDA(cudaMemcpyAsync(img_y, b->stage_iy, bytes, cudaMemcpyDeviceToHost, b->stream));
  BCUDA(cudaStreamSynchronize(b->stream));
  return SPP_OK;
}

int64_t spp_batch_kernel_launches(SppBatch* b) { return b ? b->launches : 0; }

int spp_batch_time_steps(SppBatch* b, int nsteps, double* ms) {
  if (!b || !ms) return bfail(SPP_ERR_INVALID, "NULL argument");
  if (!b->uploaded || nsteps < 0) return bfail(SPP_ERR_INVALID, "no state uploaded or bad step count");
  int rc = batch_refresh_active(b);
  if (rc != SPP_OK) return rc;
  if (b->d.n_act > 0) {  /* capture outside the timed region */
    cudaGraphExec_t exec;
    rc = batch_graph(b, nsteps >= BATCH_GRAPH_CHUNK ? BATCH_GRAPH_CHUNK : nsteps, &exec);
    if (rc == SPP_OK && nsteps % BATCH_GRAPH_CHUNK && nsteps > BATCH_GRAPH_CHUNK)
      rc = batch_graph(b, nsteps % BATCH_GRAPH_CHUNK, &exec);
    if (rc != SPP_OK) return rc;
  }
  cudaEvent_t e0, e1;
  BCUDA(cudaEventCreate(&e0));
  BCUDA(cudaEventCreate(&e1));
  cudaEventRecord(e0, b->stream);
  rc = batch_step_enqueue(b, nsteps);
  cudaEventRecord(e1, b->stream);
  cudaError_t e = cudaEventSynchronize(e1);
  float t = 0;
  if (rc == SPP_OK && e == cudaSuccess) e = cudaEventElapsedTime(&t, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc != SPP_OK) return rc;
  if (e != cudaSuccess) return bfail(SPP_ERR_CUDA, cudaGetErrorString(e));
  *ms = t;
  return SPP_OK;
}

}  // extern "C"
