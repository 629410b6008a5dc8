// Bookkeeping of a ring of bulk-copy stages for the way out of a kernel that gave up: which stages were ever armed, and
// with which parity the last copy of each one completes. (A parity wait succeeds at once on the phase before the current
// one, so waiting for "either parity" waits for nothing.) Plain code, shared with a host test.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define KDNN_RING_FN __host__ __device__ __forceinline__
#else
#define KDNN_RING_FN inline
#endif

namespace kdnn {

struct RingArmed {
  uint32_t armed = 0, parity = 0;   // bit per stage
  KDNN_RING_FN void arm(int stage, uint32_t par) {
    armed |= 1u << stage;
    parity = (parity & ~(1u << stage)) | (par << stage);
  }
};

// Waits, at most `limit` probes a stage, until the last copy of every armed stage has landed.
// try_wait(stage, parity): whether the stage's phase of that parity is complete.
template <class TryWait>
KDNN_RING_FN bool ring_drain(const RingArmed& r, int stages, uint32_t limit, TryWait try_wait) {
  bool all = true;
  for (int s = 0; s < stages; ++s) {
    if (!((r.armed >> s) & 1u)) continue;
    bool ok = false;
    for (uint32_t i = 0; i < limit && !ok; ++i) ok = try_wait(s, (r.parity >> s) & 1u);
    all = all && ok;
  }
  return all;
}

}  // namespace kdnn
