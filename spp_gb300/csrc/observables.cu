/*
 * observables.cu -- order parameters and pair statistics of a system.
 *
 * The reference computes these offline, from frames saved to disk:
 *   Compute_Order_Parameters  analyze/analyze.h:121-146  (<P>, sigma^2, error, G)
 *   Stat::Compute             analyze/statistics.h:35-54
 *   Stat::Find_Correlation_Length analyze/statistics.h:68-82
 *   Pair_Distribution         analyze/analyze.h:365-424  (body-frame histogram)
 * Here the frames come from the device: the polarization series is recorded
 * every `every` steps with the exact fixed-point heading sums, and the pair
 * histograms are built by a counting sort of the current positions into
 * cells at least as wide as the histogram's range, one thread per particle
 * walking half of its 3 x 3 cells, with per-block shared-memory histograms
 * flushed by integer atomics (the counts do not depend on the visiting
 * order).  A
 * radial g(r) is project-defined: the reference has only the body-frame
 * histogram.
 */
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>
#include "spp_internal.cuh"

namespace {

int ofail(int status, const std::string& msg) {
  spp_internal_set_error(msg.c_str());
  return status;
}

#define OCUDA(expr)                                                                        \
  do {                                                                                     \
    cudaError_t _e = (expr);                                                               \
    if (_e != cudaSuccess) return ofail(SPP_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(_e)); \
  } while (0)

/* ---------------------------------------------------------------- */
/* a counting sort of the current positions into a D x D row-major grid */
/* ---------------------------------------------------------------- */
struct Grid {
  int n, D;
  int closed;             /* a closed box: plain differences, no minimum image */
  float L, L2;
  const float4* pos;
  uint32_t *count, *start, *key, *rank, *tmp;
  float4* sorted;
};

__global__ void __launch_bounds__(SPP_BLOCK) k_obs_bin(Grid g) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  const float4 p = g.pos[i];
  const int cx = spp_cell_coord(p.x, g.L, g.L2, g.D, SPP_BIN_GEOMETRIC);
  const int cy = spp_cell_coord(p.y, g.L, g.L2, g.D, SPP_BIN_GEOMETRIC);
  const uint32_t key = (uint32_t)cy * (uint32_t)g.D + (uint32_t)cx;
  g.key[i] = key;
  g.rank[i] = atomicAdd(&g.count[key], 1u);
}

__global__ void __launch_bounds__(SPP_BLOCK) k_obs_scatter(Grid g) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  g.sorted[g.start[g.key[i]] + g.rank[i]] = g.pos[i];
}

/* Pair histograms.  Each unordered pair of particles is met once, from the
 * half of the 3 x 3 neighbourhood ahead of a particle (the rest of its own
 * cell, the cell to its right, the three cells of the row above; with at
 * least three cells per side no pair of cells meets twice), and counted as
 * its two ordered pairs: their separations are exact negatives.
 *   RADIAL    minimum-image distances below sqrt(r2max) (plain differences in
 *             a closed box), bin (int)(d / dr); the kernel counts unordered
 *             pairs and the flush doubles them
 *   body      Pair_Distribution: plain differences in the frame of the first
 *             particle's heading, both orders evaluated
 * A bin index is a monotone function of one float (d^2, t_x or t_y) with a
 * square root or divisions in it.  k_obs_edges finds by bisection, for every
 * bin, the smallest float that reaches it under that very function; a pair
 * guesses its bin with a multiplication and settles it against the edges on
 * either side, so the counts are those of the function.
 * HIST_LANES threads share a particle and take its candidates in turn (128
 * consecutive bytes).  A block keeps its histogram in shared memory,
 * `copies` words per bin side by side, a lane adding to copy lane % copies:
 * with 32 copies every lane owns a bank and no two lanes of a warp meet.
 * Blocks take chunks of particles in turn and add their bins into the global
 * counts at the end (and after every `per_flush` chunks, before a 32-bit
 * word could overflow).
 *
 * Measured at N = 262,144, unit density with flocks (one GB300, us per call,
 * sort and transfers included): g(r) to 5.0 in 50 bins 616 -> 205, body frame
 * 3 x 3 in 60 x 60 bins 897 -> 246, 1.5 x 1.5 in 10 x 10 bins 1655 -> 167; at
 * N = 4,096 232 -> 77, 169 -> 81, 134 -> 68.  Before: every ordered pair
 * evaluated, one thread per particle (a flock's particle has ten times the
 * candidates), a square root and a division per pair, one histogram per
 * block whose atomics met in few words or global atomics, and buffers
 * allocated per call.  With one thread per particle this kernel took 376, 658
 * and 385.  What bounds it: issue (distances and two edge look-ups per
 * pair). */
struct HistArgs {
  float r2max, dr;        /* RADIAL */
  float lx, ly;           /* body frame */
  int gx, gy;
  int nbins, copies, per_flush;
  int local;              /* 0: straight to the global counts (more bins than shared memory holds) */
  float inv_x, inv_y;     /* guesses: bins per unit of d, or gx / 2 / lx and gy / 2 / ly */
  const float* edges;     /* RADIAL: nbins + 1; body: gx + 1, then gy + 1 */
  int nedges;
};

__device__ __forceinline__ int radial_bin(const HistArgs& h, float d2) {
  const int b = (int)(sqrtf(d2) / h.dr);
  return b < h.nbins ? b : h.nbins - 1;
}
__device__ __forceinline__ int body_bin(int g, float l, float t) {
  const int b = (int)((float)g * ((t / l) + 1.0f) / 2.0f);
  return b < g ? b : g - 1;
}
/* floats in their order as integers */
__device__ __forceinline__ int ordered_key(float x) {
  const int i = __float_as_int(x);
  return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float ordered_float(int key) { return __int_as_float(key ^ ((key >> 31) & 0x7fffffff)); }

/* edges[b]: the smallest float of the domain whose bin is at least b
 * (-infinity for b = 0, +infinity where there is none). */
template <bool RADIAL>
__global__ void __launch_bounds__(SPP_BLOCK) k_obs_edges(HistArgs h, float* edges) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= h.nedges) return;
  const bool second = !RADIAL && e > h.gx;
  const int b = second ? e - h.gx - 1 : e;
  const int g = second ? h.gy : h.gx;
  const float l = second ? h.ly : h.lx;
  const int nb = RADIAL ? h.nbins : g;
  float edge = __int_as_float(0x7f800000);
  if (b == 0) {
    edge = -edge;
  } else if (b < nb) {
    long long lo = ordered_key(RADIAL ? 0.0f : -l), hi = (long long)ordered_key(RADIAL ? h.r2max : l) + 1;
    while (lo < hi) {   /* first key in [lo, hi) with bin >= b; hi: none */
      const long long mid = (lo + hi) >> 1;
      const float x = ordered_float((int)mid);
      if ((RADIAL ? radial_bin(h, x) : body_bin(g, l, x)) >= b) hi = mid;
      else lo = mid + 1;
    }
    if (lo <= (long long)ordered_key(RADIAL ? h.r2max : l)) edge = ordered_float((int)lo);
  }
  edges[e] = edge;
}

__device__ __forceinline__ float fast_sqrt(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

/* The bin of x between edges, from a guess (one off at most, but for sizes
 * at the ends of the float range). */
__device__ __forceinline__ int settle(int guess, int nb, float x, const float* edges) {
  int b = guess < 0 ? 0 : (guess < nb ? guess : nb - 1);
  while (x < edges[b]) --b;
  while (x >= edges[b + 1]) ++b;
  return b;
}

constexpr int HIST_THREADS = 512;
constexpr int HIST_LANES = 8;
constexpr int HIST_CHUNK = HIST_THREADS / HIST_LANES;   /* particles */

/* NEAR: the edges fit shared memory (a long thin body-frame grid's, past
 * 58,000 bins on a side, do not; they are read from global memory). */
template <bool RADIAL, bool NEAR>
__global__ void __launch_bounds__(HIST_THREADS, 2) k_obs_hist(Grid g, HistArgs h, unsigned long long* counts) {
  extern __shared__ float hist_mem[];
  const float* const edges = NEAR ? hist_mem : h.edges;                 /* [nedges] */
  uint32_t* const hist = reinterpret_cast<uint32_t*>(hist_mem + (NEAR ? h.nedges : 0));  /* [nbins][copies] */
  const int lane_copy = threadIdx.x & (h.copies - 1);
  const int words = h.local ? h.nbins * h.copies : 0;
  const int chunks = (g.n + HIST_CHUNK - 1) / HIST_CHUNK;
  for (int b = threadIdx.x; b < words; b += HIST_THREADS) hist[b] = 0u;
  if (NEAR)
    for (int b = threadIdx.x; b < h.nedges; b += HIST_THREADS) hist_mem[b] = h.edges[b];
  __syncthreads();
  auto add = [&](int b) {
    if (h.local) atomicAdd(&hist[b * h.copies + lane_copy], 1u);
    else atomicAdd(&counts[b], 1ull);
  };
  auto body = [&](float4 from, float dx, float dy) {
    const float ty = from.z * dx + from.w * dy;
    const float tx = from.w * dx - from.z * dy;
    if (fabsf(tx) < h.lx && fabsf(ty) < h.ly) {
      const int bx = settle((int)(fmaf(tx, h.inv_x, 0.5f * (float)h.gx)), h.gx, tx, edges);
      const int by = settle((int)(fmaf(ty, h.inv_y, 0.5f * (float)h.gy)), h.gy, ty, edges + h.gx + 1);
      add(bx * h.gy + by);
    }
  };
  auto pair = [&](float4 p, float4 q) {
    if (RADIAL) {
      const float dx = g.closed ? p.x - q.x : spp_min_image_f(p.x - q.x, g.L, g.L2);
      const float dy = g.closed ? p.y - q.y : spp_min_image_f(p.y - q.y, g.L, g.L2);
      const float d2 = fmaf(dx, dx, dy * dy);
      if (d2 < h.r2max) add(settle((int)(fast_sqrt(d2) * h.inv_x), h.nbins, d2, edges));
    } else {
      const float dx = q.x - p.x, dy = q.y - p.y;
      body(p, dx, dy);
      body(q, -dx, -dy);
    }
  };
  const int lr = threadIdx.x % HIST_LANES;
  int done = 0;
  for (int chunk = blockIdx.x; chunk < chunks; chunk += gridDim.x) {
    const int i = chunk * HIST_CHUNK + threadIdx.x / HIST_LANES;
    if (i < g.n) {
      const float4 p = g.sorted[i];
      const int cx = spp_cell_coord(p.x, g.L, g.L2, g.D, SPP_BIN_GEOMETRIC);
      const int cy = spp_cell_coord(p.y, g.L, g.L2, g.D, SPP_BIN_GEOMETRIC);
      const int D = g.D;
      /* ranges of candidate slots; a row's cells are contiguous */
      auto walk = [&](uint32_t s0, uint32_t s1) {
        for (uint32_t j = s0 + lr; j < s1; j += 2 * HIST_LANES) {
          const uint32_t j2 = j + HIST_LANES;
          const float4 qa = g.sorted[j], qb = g.sorted[j2 < s1 ? j2 : j];
          pair(p, qa);
          if (j2 < s1) pair(p, qb);
        }
      };
      auto first = [&](int x, int y) { return g.start[(uint32_t)y * (uint32_t)D + (uint32_t)x]; };
      auto end = [&](int x, int y) {
        const uint32_t c = (uint32_t)y * (uint32_t)D + (uint32_t)x;
        return g.start[c] + g.count[c];
      };
      const bool inner = cx > 0 && cx < D - 1;
      walk((uint32_t)i + 1u, end(inner ? cx + 1 : cx, cy));
      if (!inner) {
        if (cx < D - 1) walk(first(cx + 1, cy), end(cx + 1, cy));
        else if (RADIAL) walk(first(0, cy), end(0, cy));
      }
      /* across the boundary the body frame's plain difference exceeds the range */
      if (RADIAL || cy < D - 1) {
        const int up = cy < D - 1 ? cy + 1 : 0;
        if (inner) {
          walk(first(cx - 1, up), end(cx + 1, up));
        } else {
          walk(first(cx, up), end(cx, up));
          if (cx > 0) walk(first(cx - 1, up), end(cx - 1, up));
          else if (RADIAL) walk(first(D - 1, up), end(D - 1, up));
          if (cx < D - 1) walk(first(cx + 1, up), end(cx + 1, up));
          else if (RADIAL) walk(first(0, up), end(0, up));
        }
      }
    }
    if (!h.local || (++done < h.per_flush && chunk + (int)gridDim.x < chunks)) continue;
    done = 0;
    __syncthreads();
    for (int b = threadIdx.x; b < h.nbins; b += HIST_THREADS) {
      unsigned long long sum = 0ull;
      for (int c = 0; c < h.copies; ++c) {
        sum += hist[b * h.copies + c];
        hist[b * h.copies + c] = 0u;
      }
      if (sum) atomicAdd(&counts[b], RADIAL ? 2ull * sum : sum);
    }
    __syncthreads();
  }
}

/* Per ring: sums of x, y, x^2, y^2, xy of the unwrapped positions of its
 * beads (block 2r) and of its swimmers (block 2r + 1), in FP64 with a fixed
 * reduction tree.  Slot of particle id q: inv[q]. */
__global__ void __launch_bounds__(SPP_BLOCK) k_obs_ring_sums(DevState d, SppConsts k, int n_rings, int ring_size,
                                                             int sw_per_ring, double* sums) {
  __shared__ double red[5][SPP_BLOCK];
  const int ring = blockIdx.x >> 1, part = blockIdx.x & 1;
  const int first = part == 0 ? ring * ring_size : n_rings * ring_size + ring * sw_per_ring;
  const int count = part == 0 ? ring_size : sw_per_ring;
  double a[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  for (int q = threadIdx.x; q < count; q += blockDim.x) {
    const uint32_t slot = d.inv[first + q];
    const float4 p = d.pos[slot];
    const int2 g = d.img[slot];
    const double x = (double)p.x + (double)k.L2 * (double)g.x;
    const double y = (double)p.y + (double)k.L2 * (double)g.y;
    a[0] += x;
    a[1] += y;
    a[2] += x * x;
    a[3] += y * y;
    a[4] += x * y;
  }
  for (int c = 0; c < 5; ++c) red[c][threadIdx.x] = a[c];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w)
      for (int c = 0; c < 5; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < 5) sums[(size_t)blockIdx.x * 5 + threadIdx.x] = red[threadIdx.x][0];
}

/* Positions (unwrapped, FP64) and headings of every particle, by id: the
 * frame spp_ring_motion measures from (Save_Particles_Positions,
 * parallel/beadbox.h:315-322). */
__global__ void __launch_bounds__(SPP_BLOCK) k_obs_mark(DevState d, SppConsts k, double2* xy, float* th) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  const uint32_t id = d.id[i];
  const float4 p = d.pos[i];
  const int2 g = d.img[i];
  xy[id] = make_double2((double)p.x + (double)k.L2 * (double)g.x, (double)p.y + (double)k.L2 * (double)g.y);
  th[id] = d.theta[i];
}

/* Per ring, sums over its beads (block 2r) and its swimmers (block 2r + 1)
 * of x, y, x^2, y^2, xy, v_x, v_y, x v_y - y v_x and (swimmers) the spin,
 * with v = (r - r_marked) / elapsed and the spin the heading change folded
 * to [-pi, pi) as beadbox.h:354-356 folds it, over elapsed; FP64, fixed
 * reduction tree. */
constexpr int MOTION_SUMS = 9;
__global__ void __launch_bounds__(SPP_BLOCK) k_obs_ring_motion(DevState d, SppConsts k, int n_rings, int ring_size,
                                                               int sw_per_ring, const double2* mxy,
                                                               const float* mth, double inv_elapsed,
                                                               double* sums) {
  __shared__ double red[MOTION_SUMS][SPP_BLOCK];
  const int ring = blockIdx.x >> 1, part = blockIdx.x & 1;
  const int first = part == 0 ? ring * ring_size : n_rings * ring_size + ring * sw_per_ring;
  const int count = part == 0 ? ring_size : sw_per_ring;
  double a[MOTION_SUMS];
  for (int c = 0; c < MOTION_SUMS; ++c) a[c] = 0.0;
  const double two_pi = 6.283185307179586476925286766559;
  for (int q = threadIdx.x; q < count; q += blockDim.x) {
    const uint32_t id = (uint32_t)(first + q);
    const uint32_t slot = d.inv[id];
    const float4 p = d.pos[slot];
    const int2 g = d.img[slot];
    const double x = (double)p.x + (double)k.L2 * (double)g.x;
    const double y = (double)p.y + (double)k.L2 * (double)g.y;
    const double2 m = mxy[id];
    const double vx = (x - m.x) * inv_elapsed, vy = (y - m.y) * inv_elapsed;
    a[0] += x;
    a[1] += y;
    a[2] += x * x;
    a[3] += y * y;
    a[4] += x * y;
    a[5] += vx;
    a[6] += vy;
    a[7] += x * vy - y * vx;
    if (part == 1) {
      double dth = (double)d.theta[slot] - (double)mth[id];
      dth -= two_pi * floor(dth / two_pi);
      dth -= two_pi * floor(dth / (0.5 * two_pi));
      a[8] += dth * inv_elapsed;
    }
  }
  for (int c = 0; c < MOTION_SUMS; ++c) red[c][threadIdx.x] = a[c];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w)
      for (int c = 0; c < MOTION_SUMS; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < MOTION_SUMS) sums[(size_t)blockIdx.x * MOTION_SUMS + threadIdx.x] = red[threadIdx.x][0];
}

/* The reference's formulas (beadbox.h:402-428) from the five sums of n points. */
void shape_from_sums(const double* m, int n, double* cm_x, double* cm_y, double* xx, double* yy, double* xy,
                     double* l1, double* l2, double* rg, double* delta) {
  *cm_x = m[0] / n;
  *cm_y = m[1] / n;
  *xx = (m[2] / n) - *cm_x * *cm_x;
  *yy = (m[3] / n) - *cm_y * *cm_y;
  *xy = (m[4] / n) - *cm_x * *cm_y;
  const double root = std::sqrt((*xx - *yy) * (*xx - *yy) + 4 * *xy * *xy);
  *l1 = 0.5 * (*xx + *yy) + 0.5 * root;
  *l2 = 0.5 * (*xx + *yy) - 0.5 * root;
  *rg = std::sqrt(*xx + *yy);
  const double dl = (*l1 - *l2) / (*l1 + *l2);
  *delta = dl * dl;
}

/* Device words of one call: the system's scratch, kept, or memory of their own
 * where they are many (a series of more than half a million frames).  An
 * allocation of a few words per call costs 130 us next to a large system, whose
 * own arrays are one allocation: the few words take, and give back, a page of
 * device memory (series of 5 frames, us: 60,001 disks 346 -> 211, 400,001 552 ->
 * 412, 1M 894 -> 748). */
struct CallWords {
  unsigned long long* p = nullptr;
  bool own = false;
  ~CallWords() {
    if (own) cudaFree(p);
  }
  int take(SppSystem* s, size_t n) {
    if (n <= (1u << 20)) return spp_internal_scratch(s, n, &p);
    if (cudaMalloc((void**)&p, sizeof(*p) * n) != cudaSuccess) return ofail(SPP_ERR_ALLOC, "cudaMalloc failed");
    own = true;
    return SPP_OK;
  }
};

inline int nblk(int n) { return (n + SPP_BLOCK - 1) / SPP_BLOCK; }

int hist_edges(bool radial, const HistArgs& h) { return radial ? h.nbins + 1 : h.gx + h.gy + 2; }

/* Sorts the system's current positions into a grid of cells at least `range`
 * wide, in the system's own scratch arrays; *bins: nbins zeroed counts, then
 * room for nedges floats. */
int grid_build(SppSystem* s, double range, size_t nbins, size_t nedges, Grid* g, unsigned long long** bins, cudaStream_t* st) {
  DevState d;
  SppConsts k;
  int rc = spp_sync(s);
  if (rc != SPP_OK) return rc;
  rc = spp_internal_view(s, &d, &k, st);
  if (rc != SPP_OK) return rc;
  memset(g, 0, sizeof(*g));
  const int D = (int)std::floor(2.0 * (double)k.L / (range * 1.001));
  if (!(range > 0) || D < 3) return ofail(SPP_ERR_INVALID, "range must be in (0, 2L/3]");
  if ((double)D * D > 4.0e8) return ofail(SPP_ERR_INVALID, "range too small for the box (too many cells)");
  g->n = d.n;
  g->D = D;
  g->L = k.L;
  g->L2 = k.L2;
  g->closed = k.closed;
  g->pos = d.pos;
  g->key = d.key;
  g->rank = d.rank;
  g->sorted = d.pos_alt;
  const size_t nc = (size_t)D * D;
  rc = spp_internal_obs_space(s, nc, nbins + (nedges + 1) / 2, &g->count, &g->start, &g->tmp, bins);
  if (rc != SPP_OK) return rc;
  OCUDA(cudaMemsetAsync(g->count, 0, sizeof(uint32_t) * nc, *st));
  OCUDA(cudaMemsetAsync(*bins, 0, sizeof(unsigned long long) * nbins, *st));
  k_obs_bin<<<nblk(g->n), SPP_BLOCK, 0, *st>>>(*g);
  launch_scan_u32(g->count, (uint32_t)nc, g->tmp, g->start, *st, nullptr);
  k_obs_scatter<<<nblk(g->n), SPP_BLOCK, 0, *st>>>(*g);
  OCUDA(cudaGetLastError());
  spp_internal_count_launches(s, 4);
  return SPP_OK;
}

/* The histogram of the grid's pairs into bins, with smem bytes of shared
 * memory per block. */
template <bool RADIAL, bool NEAR>
int launch_hist(const Grid& g, const HistArgs& h, unsigned long long* bins, int sms, int most, size_t smem,
                cudaStream_t st) {
  OCUDA(cudaFuncSetAttribute(k_obs_hist<RADIAL, NEAR>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
  int per_sm = 1;
  OCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_obs_hist<RADIAL, NEAR>, HIST_THREADS, smem));
  const int chunks = (g.n + HIST_CHUNK - 1) / HIST_CHUNK;
  const int blocks = std::min(chunks, sms * std::max(per_sm, 1));
  k_obs_hist<RADIAL, NEAR><<<blocks, HIST_THREADS, smem, st>>>(g, h, bins);
  return SPP_OK;
}

/* The histogram of the grid's pairs into counts (host). */
template <bool RADIAL>
int run_hist(SppSystem* s, const Grid& g, HistArgs h, unsigned long long* bins, uint64_t* counts, cudaStream_t st) {
  int dev = 0, sms = 0, most = 0;
  OCUDA(cudaGetDevice(&dev));
  OCUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  OCUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  h.nedges = hist_edges(RADIAL, h);
  h.edges = reinterpret_cast<float*>(bins + h.nbins);
  /* as many copies of the histogram as fit a third of an SM's shared memory
   * (two blocks per SM); one copy up to all of it; else global atomics */
  const size_t one = sizeof(uint32_t) * (size_t)h.nbins, fixed = sizeof(float) * (size_t)h.nedges;
  h.local = one + fixed <= (size_t)most;
  h.copies = 1;
  while (h.local && h.copies < 32 && 2 * h.copies * one <= (size_t)most / 3) h.copies *= 2;
  /* a chunk adds at most HIST_CHUNK x 2 n to a bin */
  const double chunk_most = 2.0 * HIST_CHUNK * (double)g.n;
  if (chunk_most >= 4294967295.0) h.local = 0;
  h.per_flush = (int)std::fmin(1e6, std::floor(4294967295.0 / chunk_most));
  if (!h.local) h.copies = 1;
  const bool near = fixed <= (size_t)most;   /* a radial histogram's edges always are */
  const size_t smem = (near ? fixed : 0) + (h.local ? h.copies * one : 0);
  k_obs_edges<RADIAL><<<nblk(h.nedges), SPP_BLOCK, 0, st>>>(h, const_cast<float*>(h.edges));
  const int rc = RADIAL || near ? launch_hist<RADIAL, true>(g, h, bins, sms, most, smem, st)
                                : launch_hist<false, false>(g, h, bins, sms, most, smem, st);
  if (rc != SPP_OK) return rc;
  spp_internal_count_launches(s, 2);
  OCUDA(cudaGetLastError());
  OCUDA(cudaMemcpyAsync(counts, bins, sizeof(uint64_t) * (size_t)h.nbins, cudaMemcpyDeviceToHost, st));
  OCUDA(cudaStreamSynchronize(st));
  if (RADIAL && !h.local)   /* counted straight into the global bins, once per unordered pair */
    for (int b = 0; b < h.nbins; ++b) counts[b] *= 2;
  return SPP_OK;
}

/* Autocorrelation length as Stat::Find_Correlation_Length computes it: the
 * first lag tau < T/2 at which the normalised autocorrelation, each term
 * divided by (T - tau) before it is added, falls below 0.01 (T/2 - 1 when
 * none does; 0 when the series is constant). */
double correlation_length(const double* x, int T, double mean, double variance) {
  double corr_len = 0.0;
  for (int tau = 0; tau < T / 2; ++tau) {
    double c = 0.0;
    for (int i = 0; i < T - tau; ++i) c += (x[i] - mean) * (x[i + tau] - mean) / (double)(T - tau);
    c /= variance;
    corr_len = (double)tau;
    if (c < 0.01) break;
  }
  return corr_len;
}

}  // namespace

extern "C" {

int spp_order_parameters(const double* p, int T, double area, SppOrderStats* out) {
  if (!p || !out || T < 2) return ofail(SPP_ERR_INVALID, "need a series of at least 2 samples");
  memset(out, 0, sizeof(*out));
  double mn = p[0], mx = p[0], sum = 0.0, sq = 0.0, sum4 = 0.0;
  for (int i = 0; i < T; ++i) {
    if (!std::isfinite(p[i])) return ofail(SPP_ERR_NUMERIC, "non-finite sample");
    mn = p[i] < mn ? p[i] : mn;
    mx = p[i] > mx ? p[i] : mx;
    sum += p[i];
    sq += p[i] * p[i];
    const double p2 = p[i] * p[i];
    sum4 += p2 * p2;
  }
  out->samples = T;
  out->min = mn;
  out->max = mx;
  out->mean = sum / T;
  out->mean_square = sq / T;
  out->variance = out->mean_square - out->mean * out->mean;
  out->std = std::sqrt(out->variance);
  out->corr_len = correlation_length(p, T, out->mean, out->variance);
  out->error = std::sqrt(out->variance * out->corr_len / T);
  out->sigma2 = out->variance * area;
  out->p4_mean = sum4 / T;
  if (out->mean_square > 0) {
    out->binder = 1.0 - out->p4_mean / (3.0 * out->mean_square * out->mean_square);
    out->binder_reference = 1.0 - out->p4_mean / (3.0 * out->mean_square);
  }
  return SPP_OK;
}

int spp_polarization_series(SppSystem* s, int nframes, int every, double* p, double* px, double* py) {
  if (!s || !p || nframes < 1 || every < 1) return ofail(SPP_ERR_INVALID, "bad arguments");
  DevState d;
  SppConsts k;
  cudaStream_t st;
  int rc = spp_internal_view(s, &d, &k, &st);
  if (rc != SPP_OK) return rc;
  CallWords words;
  rc = words.take(s, 2 * (size_t)nframes);
  if (rc != SPP_OK) return rc;
  unsigned long long* const sums = words.p;
  std::vector<long long> host(2 * (size_t)nframes);
  cudaError_t e = cudaMemsetAsync(sums, 0, sizeof(unsigned long long) * 2 * (size_t)nframes, st);
  /* the Verlet-list models may freeze on a full neighbour list; their frames
   * wait for the steps (re-run by spp_sync) before P is read.  The Vicsek
   * models have no list: their frames queue up without host round trips. */
  const bool listed = k.model == SPP_MODEL_ABP || k.model == SPP_MODEL_CONTINUOUS || k.model == SPP_MODEL_BEADS;
  int whole = 1;   /* 0: every frame in one resident run */
  if (e == cudaSuccess) {
    whole = spp_internal_series(s, nframes, every, sums);
    if (whole < 0) rc = whole == -1 ? SPP_ERR_INVALID : SPP_ERR_CUDA;
  }
  for (int f = 0; whole > 0 && f < nframes && rc == SPP_OK && e == cudaSuccess; ++f) {
    rc = spp_step(s, every);
    if (rc == SPP_OK && listed) rc = spp_sync(s);
    if (rc == SPP_OK) {
      rc = spp_internal_view(s, &d, &k, &st);
      launch_polarization_into(d, sums + 2 * (size_t)f, st);
      spp_internal_count_launches(s, 1);
      e = cudaGetLastError();
    }
  }
  if (rc == SPP_OK && e == cudaSuccess)
    e = cudaMemcpyAsync(host.data(), sums, sizeof(long long) * host.size(), cudaMemcpyDeviceToHost, st);
  if (rc == SPP_OK && e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (rc == SPP_OK && e == cudaSuccess && !listed) rc = spp_sync(s);   /* device-side status */
  if (rc != SPP_OK) return rc;
  if (e != cudaSuccess) return ofail(SPP_ERR_CUDA, cudaGetErrorString(e));
  const double inv = 1.0 / 134217728.0; /* fixed-point units of 2^-27 */
  for (int f = 0; f < nframes; ++f) {
    const double ax = (double)host[2 * (size_t)f] * inv / d.n;
    const double ay = (double)host[2 * (size_t)f + 1] * inv / d.n;
    p[f] = std::sqrt(ax * ax + ay * ay);
    if (px) px[f] = ax;
    if (py) py[f] = ay;
  }
  return SPP_OK;
}

int spp_radial_distribution(SppSystem* s, double r_max, int nbins, uint64_t* counts) {
  if (!s || !counts || nbins < 1 || nbins > 4096) return ofail(SPP_ERR_INVALID, "bad arguments");
  Grid g;
  cudaStream_t st;
  unsigned long long* bins = nullptr;
  HistArgs h = {};
  const float rm = (float)r_max;
  h.r2max = rm * rm;
  h.dr = rm / (float)nbins;
  h.nbins = nbins;
  h.inv_x = 1.0f / h.dr;
  int rc = grid_build(s, r_max, (size_t)nbins, (size_t)hist_edges(true, h), &g, &bins, &st);
  if (rc != SPP_OK) return rc;
  return run_hist<true>(s, g, h, bins, counts, st);
}

int spp_pair_distribution(SppSystem* s, double lx, double ly, int gx, int gy, uint64_t* counts) {
  if (!s || !counts || gx < 1 || gy < 1 || (int64_t)gx * gy > 65536 || !(lx > 0) || !(ly > 0))
    return ofail(SPP_ERR_INVALID, "bad arguments");
  Grid g;
  cudaStream_t st;
  unsigned long long* bins = nullptr;
  HistArgs h = {};
  h.lx = (float)lx;
  h.ly = (float)ly;
  h.gx = gx;
  h.gy = gy;
  h.nbins = gx * gy;
  h.inv_x = 0.5f * (float)gx / h.lx;
  h.inv_y = 0.5f * (float)gy / h.ly;
  int rc = grid_build(s, std::sqrt(lx * lx + ly * ly), (size_t)gx * gy, (size_t)hist_edges(false, h), &g, &bins, &st);
  if (rc != SPP_OK) return rc;
  return run_hist<false>(s, g, h, bins, counts, st);
}

int spp_ring_shapes(SppSystem* s, SppRingShape* out, int n_rings) {
  if (!s || !out) return ofail(SPP_ERR_INVALID, "NULL argument");
  int rc = spp_sync(s);
  if (rc != SPP_OK) return rc;
  DevState d;
  SppConsts k;
  cudaStream_t st;
  rc = spp_internal_view(s, &d, &k, &st);
  if (rc != SPP_OK) return rc;
  if (k.model != SPP_MODEL_BEADS || k.n_beads <= 0 || k.ring_size <= 0)
    return ofail(SPP_ERR_INVALID, "ring shapes need a bead model with rings");
  const int nr = k.n_beads / k.ring_size;
  if (n_rings != nr) return ofail(SPP_ERR_INVALID, "n_rings differs from the system's ring count");
  const int sw = (d.n - k.n_beads) / nr;
  CallWords words;
  rc = words.take(s, 10 * (size_t)nr);
  if (rc != SPP_OK) return rc;
  double* const sums = reinterpret_cast<double*>(words.p);
  k_obs_ring_sums<<<2 * nr, SPP_BLOCK, 0, st>>>(d, k, nr, k.ring_size, sw, sums);
  spp_internal_count_launches(s, 1);
  std::vector<double> h(10 * (size_t)nr);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), sums, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return ofail(SPP_ERR_CUDA, std::string("ring shapes: ") + cudaGetErrorString(e));
  for (int r = 0; r < nr; ++r) {
    SppRingShape& o = out[r];
    memset(&o, 0, sizeof(o));
    shape_from_sums(&h[10 * (size_t)r], k.ring_size, &o.mb_cm_x, &o.mb_cm_y, &o.mb_xx, &o.mb_yy, &o.mb_xy,
                    &o.mb_lambda1, &o.mb_lambda2, &o.mb_Rg, &o.mb_Delta);
    if (sw > 0)
      shape_from_sums(&h[10 * (size_t)r + 5], sw, &o.sw_cm_x, &o.sw_cm_y, &o.sw_xx, &o.sw_yy, &o.sw_xy,
                      &o.sw_lambda1, &o.sw_lambda2, &o.sw_Rg, &o.sw_Delta);
  }
  return SPP_OK;
}

int spp_ring_motion_mark(SppSystem* s) {
  if (!s) return ofail(SPP_ERR_INVALID, "NULL argument");
  int rc = spp_sync(s);
  if (rc != SPP_OK) return rc;
  DevState d;
  SppConsts k;
  cudaStream_t st;
  rc = spp_internal_view(s, &d, &k, &st);
  if (rc != SPP_OK) return rc;
  double2* xy;
  float* th;
  int64_t* step;
  rc = spp_internal_mark(s, &xy, &th, &step);
  if (rc != SPP_OK) return rc;
  k_obs_mark<<<nblk(d.n), SPP_BLOCK, 0, st>>>(d, k, xy, th);
  spp_internal_count_launches(s, 1);
  OCUDA(cudaGetLastError());
  const int64_t now = spp_internal_step(s);   /* waits for the stream */
  if (now < 0) return ofail(SPP_ERR_CUDA, "ring motion: reading the step counter failed");
  *step = now;
  return SPP_OK;
}

int spp_ring_motion(SppSystem* s, SppRingMotion* out, int n_rings) {
  if (!s || !out) return ofail(SPP_ERR_INVALID, "NULL argument");
  int rc = spp_sync(s);
  if (rc != SPP_OK) return rc;
  DevState d;
  SppConsts k;
  cudaStream_t st;
  rc = spp_internal_view(s, &d, &k, &st);
  if (rc != SPP_OK) return rc;
  if (k.model != SPP_MODEL_BEADS || k.n_beads <= 0 || k.ring_size <= 0)
    return ofail(SPP_ERR_INVALID, "ring motion needs a bead model with rings");
  const int nr = k.n_beads / k.ring_size;
  if (n_rings != nr) return ofail(SPP_ERR_INVALID, "n_rings differs from the system's ring count");
  double2* xy;
  float* th;
  int64_t* mark;
  rc = spp_internal_mark(s, &xy, &th, &mark);
  if (rc != SPP_OK) return rc;
  if (*mark < 0) return ofail(SPP_ERR_INVALID, "no frame marked: call spp_ring_motion_mark first");
  const int64_t now = spp_internal_step(s);
  if (now < 0) return ofail(SPP_ERR_CUDA, "ring motion: reading the step counter failed");
  if (now <= *mark) return ofail(SPP_ERR_INVALID, "no step taken since the marked frame");
  const double elapsed = (double)(now - *mark) * spp_internal_dt(s);
  const int sw = (d.n - k.n_beads) / nr;
  CallWords words;
  rc = words.take(s, 2 * MOTION_SUMS * (size_t)nr);
  if (rc != SPP_OK) return rc;
  double* const sums = reinterpret_cast<double*>(words.p);
  k_obs_ring_motion<<<2 * nr, SPP_BLOCK, 0, st>>>(d, k, nr, k.ring_size, sw, xy, th, 1.0 / elapsed, sums);
  spp_internal_count_launches(s, 1);
  std::vector<double> h(2 * MOTION_SUMS * (size_t)nr);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), sums, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return ofail(SPP_ERR_CUDA, std::string("ring motion: ") + cudaGetErrorString(e));
  for (int r = 0; r < nr; ++r) {
    /* Compute_All_Variables, parallel/beadbox.h:385-428 */
    const double* m = &h[2 * MOTION_SUMS * (size_t)r];
    const double* w = m + MOTION_SUMS;
    const double Nm = k.ring_size, Ns = sw;
    SppRingMotion& o = out[r];
    memset(&o, 0, sizeof(o));
    const double mcx = m[0] / Nm, mcy = m[1] / Nm;
    o.mb_v_cm_x = m[5] / Nm;
    o.mb_v_cm_y = m[6] / Nm;
    const double mxx = m[2] / Nm - mcx * mcx, myy = m[3] / Nm - mcy * mcy;
    o.mb_l = m[7] / Nm - mcx * o.mb_v_cm_y + mcy * o.mb_v_cm_x;
    o.mb_omega = o.mb_l / (mxx + myy);
    if (sw > 0) {
      const double scx = w[0] / Ns, scy = w[1] / Ns;
      o.sw_v_cm_x = w[5] / Ns;
      o.sw_v_cm_y = w[6] / Ns;
      const double sxx = w[2] / Ns - scx * scx, syy = w[3] / Ns - scy * scy;
      o.sw_l = w[7] / Ns - scx * o.mb_v_cm_y + scy * o.mb_v_cm_x - mcx * o.sw_v_cm_y + mcy * o.sw_v_cm_x +
               mcx * o.mb_v_cm_y - mcy * o.mb_v_cm_x;
      o.sw_spin = w[8] / Ns;
      const double dcx = mcx - scx, dcy = mcy - scy;
      o.sw_omega = o.sw_l / (sxx + syy + dcx * dcx + dcy * dcy);
    }
  }
  /* the current frame becomes the marked one (Save_Particles_Positions at
   * the end of Compute_All_Variables) */
  k_obs_mark<<<nblk(d.n), SPP_BLOCK, 0, st>>>(d, k, xy, th);
  spp_internal_count_launches(s, 1);
  OCUDA(cudaGetLastError());
  OCUDA(cudaStreamSynchronize(st));
  *mark = now;
  return SPP_OK;
}

}  // extern "C"
