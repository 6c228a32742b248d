/*
 * spp_internal.cuh -- device data layout and kernel entry points.
 *
 * HBM layout of one system (structure of arrays, all in cell order: particles
 * are counting-sorted by the Morton key of their cell at every list rebuild):
 *   pos     float4 (x, y, cos theta, sin theta)  read by neighbours, 16 B
 *   half    float4 stage state of Runge-Kutta stages (RK4 ping-pongs with half2)
 *   theta   float, img int2 (box crossings), id uint32 (slot -> particle id)
 *   kacc    float4 RK4 slope accumulator (fx, fy, tau, -)
 *   ref     float2 positions at the last neighbour-list build
 *   nbr     int32 [cap][n] neighbour slots, column-major so that a warp's
 *           32 consecutive particles read 128 contiguous bytes per list slot
 *   nn      int32 list lengths
 *   cell_count / cell_start  uint32 per Morton key
 * A small control block (Ctl) in device memory carries the step counter and
 * the device-side rebuild decision, so captured graphs replay without host
 * round trips.
 */
#ifndef SPP_INTERNAL_CUH
#define SPP_INTERNAL_CUH

#include <cuda_runtime.h>
#include <stdint.h>
#include "spp_parts.h"
#include "spp_physics.h"

#define SPP_BLOCK 256

struct Ctl {
  uint32_t step;          /* absolute step index (Philox counter word) */
  uint32_t dmax2_bits;    /* max squared displacement since the last build (float bits) */
  uint32_t blocks_done;   /* last-block detection */
  uint32_t need_rebuild;  /* decision of the last step */
  uint32_t list_need;     /* largest neighbour count met by a build (overflow if > cap) */
  uint32_t fx_overflow;   /* a pair term left the fixed-point range */
  uint32_t max_nn;        /* largest list length of the last build */
  uint32_t n_rebuilds;
  uint32_t frozen;        /* set on list overflow: later stages skip until the host recovers */
  uint32_t smax2_bits;    /* max squared displacement during the current step (float bits) */
  uint32_t late_rebuilds; /* rebuilds decided after some particle had already moved > skin/2 */
  uint32_t bad_nonfinite; /* smallest index of an uploaded particle with a non-finite value (or ~0) */
  uint32_t bad_range;     /* smallest index of an uploaded position outside [-L, L) (or ~0) */
  uint32_t long_n;        /* lists longer than the in-block sort queued by the last build */
  uint32_t bad_index;     /* SPP_CHECKED builds: a kernel met an index out of range */
  uint32_t bulk_timeouts; /* warps whose bulk copy of list rows did not arrive in time (they read global memory) */
  /* resident runs (kernels_run.cu): largest squared displacements of step t
   * in slot t % 3, blocks that have left the launch, a barrier wait that
   * gave up, and the barrier's arrival count on a cache line of its own */
  uint32_t run_disp[3], run_step[3];
  uint32_t run_exit;
  uint32_t run_timeout;
  uint32_t run_sorted;    /* step at which a resident Vicsek run last put its owners in cell order */
  uint32_t pad0[31];
  uint32_t run_bar;
  uint32_t pad1[31];
};

/* SPP_CHECKED builds check every list, cell and slot index a hot kernel
 * uses; an index out of [0, bound) sets Ctl.bad_index (the next sync
 * returns SPP_ERR_BOUNDS) and the caller skips the access.  Without
 * SPP_CHECKED the check is the constant true. */
#ifdef SPP_CHECKED
__device__ __forceinline__ bool spp_index_ok(Ctl* ctl, long long idx, long long bound) {
  if (idx >= 0 && idx < bound) return true;
  atomicOr(&ctl->bad_index, 1u);
  return false;
}
#else
__device__ __forceinline__ bool spp_index_ok(Ctl*, long long, long long) { return true; }
#endif

struct DevState {
  int n;
  int cap;
  int D;                  /* cells per side */
  int morton_bits;
  uint32_t n_keys;        /* 4^morton_bits */
  float4* pos;
  float4* half;
  float4* half2;
  float* theta;
  int2* img;
  uint32_t* id;
  uint32_t* inv;          /* particle id -> slot (ring neighbours of membrane beads) */
  float4* kacc;
  float* dth;             /* rotational noise of the current step (multi-stage integrators) */
  float2* ref;
  float4* pos_alt;
  float* theta_alt;
  int2* img_alt;
  uint32_t* id_alt;
  uint32_t* key;
  uint32_t* rank;
  uint32_t* cell_count;
  uint32_t* cell_start;
  uint32_t* scan_tmp;     /* block sums of the scan */
  int32_t* nbr;
  int32_t* nn;
  int32_t* long_q;        /* particles whose list k_sort_long orders (n entries) */
  unsigned long long* nn_lanes; /* list entries per id % 4, 16 bits each (lanes > 1), else NULL */
  int32_t* tumble;        /* run-and-tumble state by particle id (SPP_NOISE_TUMBLE), else NULL */
  Ctl* ctl;
  double* red;            /* reduction scratch (polarization) */
  uint32_t* run_sums;     /* per-block cell totals of a resident run's rebuild (RUN_MAX_BLOCKS) */
};

/* api.cu: the device state, constants and stream of an uploaded system
 * (observables.cu), and the host-launch counter */
int spp_internal_view(SppSystem* s, DevState* d, SppConsts* k, cudaStream_t* st);
void spp_internal_count_launches(SppSystem* s, int n);
/* api.cu: the marked-frame buffers of spp_ring_motion (n entries each, by
 * particle id; allocated on first use) and the mark's step (-1: none) */
int spp_internal_mark(SppSystem* s, double2** xy, float** th, int64_t** step);
/* api.cu: scratch of the pair statistics, kept with the system: counts and
 * starts of `cells` cells with the scan's block sums (the rebuild's own
 * arrays where they are large enough), and `bins` 64-bit counts */
int spp_internal_obs_space(SppSystem* s, size_t cells, size_t bins, uint32_t** count, uint32_t** start, uint32_t** tmp,
                           unsigned long long** counts);
/* api.cu: `words` 64-bit words of the same scratch, for one call's sums */
int spp_internal_scratch(SppSystem* s, size_t words, unsigned long long** out);
/* api.cu: nframes x every steps of a resident Vicsek run with the heading
 * sums of every frame; 1: not such a system, < 0: error (message set) */
int spp_internal_series(SppSystem* s, int nframes, int every, unsigned long long* sums);
/* noalloc.cu: unique id of the calling thread's current context; false if
 * there is none (the runtime has not made one current on this thread yet) or
 * the driver does not offer the entry points */
bool spp_internal_context(unsigned long long* id);
/* api.cu: the absolute step counter (waits for the stream); -1 on error */
int64_t spp_internal_step(SppSystem* s);
/* api.cu: the time step as given (double) */
double spp_internal_dt(SppSystem* s);

/* api.cu: sets the message spp_last_error() returns on the calling thread */
void spp_internal_set_error(const char* msg);

/* kernels_cells.cu */
void launch_bin_count(const SppConsts& k, const DevState& d, cudaStream_t s, int64_t* launches);
void launch_scan(const DevState& d, cudaStream_t s, int64_t* launches);
/* exclusive scan of n counts; block_tmp holds ceil(n / 4096) entries; counts
 * and out start on 16-byte boundaries */
void launch_scan_u32(uint32_t* counts, uint32_t n, uint32_t* block_tmp, uint32_t* out, cudaStream_t s,
                     int64_t* launches);
/* the same for a step's cell counts: out has one entry more (the total), and
 * the counts are cleared as they are read */
void launch_scan_counts(uint32_t* counts, uint32_t n, uint32_t* block_tmp, uint32_t* out, cudaStream_t s);
uint32_t scan_max_elements();
void launch_scatter(const DevState& d, bool vicsek, cudaStream_t s, int64_t* launches);
void launch_build_list(const SppConsts& k, const DevState& d, int with_list, cudaStream_t s,
                       int64_t* launches);
void launch_pairs_count(const SppConsts& k, const DevState& d, float r2, unsigned long long* counter,
                        int32_t* pi, int32_t* pj, long long cap, cudaStream_t s);
void launch_cells(const SppConsts& k, const DevState& d, int D, int rule, int32_t* cx, int32_t* cy,
                  cudaStream_t s);
/* Also checks the inputs (finite, positions in [-L, L)) into Ctl::bad_*;
 * img_xy (may be NULL): 2n int32 box-crossing counters, x then y. */
void launch_init_state(const SppConsts& k, const DevState& d, const float* x, const float* y,
                       const float* th, const int32_t* img_xy, cudaStream_t s);
/* img_xy: 2n int32, x counters then y counters (particle-id order) */
void launch_gather_state(const SppConsts& k, const DevState& d, float* x, float* y, float* th,
                         int32_t* img_xy, cudaStream_t s);

/* kernels_step.cu */
void prepare_abp_stage();
void launch_abp_stage(const SppConsts& k, const DevState& d, int stage, int nstages,
                      cudaGraphConditionalHandle cond, int use_cond, cudaStream_t s,
                      int64_t* launches);
/* kernels_run.cu: nsteps whole steps of a Verlet-list system in one
 * cooperative launch.  plan_run: whether the system fits (every thread of
 * its neighbour sums resident at once) and the launch shape. */
struct RunPlan {
  int blocks, threads;    /* 0: the system does not fit */
  int per_sm;             /* blocks per SM the kernel is compiled for (1 or 2) */
};
bool plan_run(const SppConsts& k, const DevState& d, RunPlan* plan);
int launch_run(const SppConsts& k, const DevState& d, const RunPlan& plan, int nstages, int nsteps, cudaStream_t s);
/* kernels_vrun.cu: the same for the discrete Vicsek models.  every > 0: the
 * fixed-point heading sums after the steps first, first + every, ... are added
 * into sums (two words per frame, zeroed by the caller). */
struct VrunPlan {
  int blocks, threads;    /* 0 blocks: the system does not fit */
  int lanes, per_sm;
  uint32_t cells;         /* D * D, rounded up to a multiple of 4 */
  int cap;                /* places per cell bucket */
};
struct VrunBufs {
  uint32_t* count[3];
  uint32_t* full;         /* [3], then the two words that a launch leaves to the next: */
  uint32_t* dirty;        /* not 0: counts and full are to be cleared first (new buffers, a barrier that gave up) */
  uint32_t* phase;        /* which of the counts the next launch starts with */
  float4* bucket[2];      /* [cells][cap] */
  float* bucket_th[2];    /* headings, angle rule only */
  uint32_t cells;
  int cap;
};
bool plan_vrun(const SppConsts& k, const DevState& d, VrunPlan* plan);
int launch_vrun(const SppConsts& k, const DevState& d, const VrunPlan& plan, const VrunBufs& vb, int nsteps, int first,
                int every, unsigned long long* sums, cudaStream_t s);
void launch_vicsek_step(const SppConsts& k, const DevState& d, cudaStream_t s, int64_t* launches);
void launch_polarization(const DevState& d, cudaStream_t s);
/* the two fixed-point heading sums added into sums[0..1] (zeroed by the caller) */
void launch_polarization_into(const DevState& d, unsigned long long* sums, cudaStream_t s);

#endif
