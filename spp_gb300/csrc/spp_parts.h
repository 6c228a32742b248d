/* spp_parts.h -- how the host cuts the steps of a call into resident launches
 * (api.cu; kernels_run.cu, kernels_vrun.cu and kernels_lrun.cu run one). */
#ifndef SPP_PARTS_H
#define SPP_PARTS_H

#include "spp_physics.h"

/* Steps of one resident launch at most, however far apart the events (frames,
 * renormalisations) of the call are.
 * A launch that fills the GPU lets no other such launch in before it ends, so
 * its length is how long a call on another handle may wait (two steps of a
 * Vicsek system of 50,001 beside a long run of 16,384 disks: 120 to 140 ms with
 * launches of 16,384 steps, 4.4 with 512, 2.2 with 256, 1.1 with 128), and its
 * start is what a long call pays for it (us per step with 16,384 / 512 / 256 /
 * 128: 4,096 Vicsek particles 5.42 / 5.44 / 5.46 / 5.49, 16,384 disks 8.44 /
 * 8.45 / 8.47 / 8.49).
 * A block arrives at the grid barrier at
 * most RUN_ARRIVALS times per step (four stages, six in a rebuild, one
 * before a renormalisation, four in it and one after), and a launch has at most
 * RUN_MAX_BLOCKS blocks: the 32-bit arrival count, compared as it stands,
 * cannot wrap. */
#define RUN_CHUNK 256
#define RUN_MAX_BLOCKS 1024
#define RUN_ARRIVALS 16
static_assert((int64_t)RUN_CHUNK * RUN_ARRIVALS * RUN_MAX_BLOCKS < ((int64_t)1 << 31), "grid barrier's arrival count");

/* Events at the steps first, first + every, ...: how many up to step x, and
 * how many steps from there to the next. */
SPP_HD int spp_events_upto(int x, int first, int every) { return x < first ? 0 : 1 + (x - first) / every; }
SPP_HD int spp_next_event(int x, int first, int every) {
  return x < first ? first - x : every - (x - first) % every;
}

/* A resident Vicsek run puts its owners in cell order RUN_SORT_STEPS steps after
 * the last time, counted over calls (Ctl.run_sorted): calls of 16 steps that
 * counted for themselves would keep the order of the upload for ever. */
#define RUN_SORT_STEPS 16u
SPP_HD bool spp_sort_due(uint32_t step, uint32_t sorted) { return step - sorted >= RUN_SORT_STEPS; }

struct RunPart {
  int steps;    /* of this launch */
  int first;    /* its step that ends with the first event (may lie beyond it); 0: no events */
  int events;   /* events within it */
  bool last;    /* the call ends with it */
};

/* nsteps steps with an event after every `every` (0: none): f(part) for every
 * launch in turn, until one does not return 0. */
template <class F>
int spp_for_parts(int64_t nsteps, int every, F f) {
  int first = every;
  while (nsteps > 0) {
    RunPart q;
    q.steps = nsteps > RUN_CHUNK ? RUN_CHUNK : (int)nsteps;
    q.first = first;
    q.events = every > 0 ? spp_events_upto(q.steps, first, every) : 0;
    q.last = nsteps == q.steps;
    const int rc = f(q);
    if (rc != 0) return rc;
    if (every > 0) first = spp_next_event(q.steps, first, every);
    nsteps -= q.steps;
  }
  return 0;
}

#endif
