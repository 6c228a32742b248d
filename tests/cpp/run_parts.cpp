// The cutting of calls into resident launches (spp_parts.h), for ctypes.
#include "../../spp_gb300/csrc/spp_parts.h"

extern "C" {

int run_chunk() { return RUN_CHUNK; }
int run_arrivals() { return RUN_ARRIVALS; }
int run_max_blocks() { return RUN_MAX_BLOCKS; }

int sort_steps() { return (int)RUN_SORT_STEPS; }
int sort_due(uint32_t step, uint32_t sorted) { return spp_sort_due(step, sorted); }

// out: four words per launch (steps, first, events, last); the launches, or -1
// once there are more than `room`.
int parts(int64_t nsteps, int every, int32_t* out, int room) {
  int n = 0;
  const int rc = spp_for_parts(nsteps, every, [&](const RunPart& q) {
    if (n == room) return 1;
    const int32_t row[4] = {q.steps, q.first, q.events, q.last};
    for (int c = 0; c < 4; ++c) out[4 * n + c] = row[c];
    ++n;
    return 0;
  });
  return rc ? -1 : n;
}
}
