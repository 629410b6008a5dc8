// Host model of the ring bookkeeping of csrc/kdnn_ring.cuh: a barrier per stage with the phase rule of an mbarrier (a
// parity wait succeeds when the phase of that parity is the one before the current one), copies that land a few probes
// late. The drain has to return after the last copy of every armed stage has landed, not before, and within its limit.
#include <stdio.h>

#include <initializer_list>

#include "../../dnn-for-kokkos_b200/csrc/kdnn_ring.cuh"

struct Barrier {
  uint32_t phase = 0;     // phases completed
  int in_flight = -1;     // probes until the armed copy lands, -1: none
  void land() { if (in_flight >= 0) { in_flight = -1; ++phase; } }
  bool try_wait(uint32_t parity) {
    if (in_flight > 0) --in_flight;
    else if (in_flight == 0) land();
    return ((phase ^ parity) & 1u) != 0;   // the phase of that parity is behind us
  }
};

// the tcgen05 kernels' loaders: stage and phase from a sequence number, and from a stage counter with a toggling phase
static int run(int stages, int armed_copies, int late, bool toggling) {
  Barrier bar[8];
  kdnn::RingArmed ring;
  int s = 0;
  uint32_t ph = 1;
  for (int seq = 0; seq < armed_copies; ++seq) {
    const int st = toggling ? s : seq % stages;
    bar[st].land();                                    // the consumer's wait and release of the copy before
    ring.arm(st, toggling ? ph ^ 1u : (static_cast<uint32_t>(seq / stages) & 1u));
    bar[st].in_flight = late + st;
    if (++s == stages) { s = 0; ph ^= 1u; }
  }
  const bool all = kdnn::ring_drain(ring, stages, 64, [&](int st, uint32_t parity) { return bar[st].try_wait(parity); });
  for (int st = 0; st < stages; ++st)
    if (bar[st].in_flight >= 0 && late + st < 60) return printf("stages %d, copies %d, late %d: stage %d still in flight\n", stages, armed_copies, late, st), 1;
  if (all != (armed_copies == 0 || late < 50)) return printf("stages %d, copies %d, late %d: drained %d\n", stages, armed_copies, late, all), 1;
  return 0;
}

int main() {
  int bad = 0;
  for (int stages = 2; stages <= 8; ++stages)
    for (int copies = 0; copies <= 4 * stages + 1; ++copies)
      for (int late : {0, 1, 7, 100})
        for (int t = 0; t < 2; ++t) bad += run(stages, copies, late, t != 0);
  // what waiting for either parity does: it returns with the copy in flight
  Barrier b;
  b.in_flight = 5;
  if (!(b.try_wait(0) || b.try_wait(1)) || b.in_flight < 0) { printf("model\n"); ++bad; }
  puts(bad ? "FAIL" : "ok");
  return bad != 0;
}
