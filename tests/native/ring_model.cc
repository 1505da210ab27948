// Model of a producer's ring of stages that is left early (csrc/common/ring.h): whatever was issued and whatever of the last
// lap is still in flight, the wait for a stage blocks exactly while its last load has not landed.
#include <cstdint>
#include <cstdio>

#include "ring.h"

// what mbarrier.try_wait.parity answers for a barrier that has completed `phases` phases
static bool try_wait(int phases, uint32_t parity) { return (static_cast<uint32_t>(phases) & 1) != parity; }

int main() {
  long checked = 0, wrong = 0;
  for (int stages = 1; stages <= 8; ++stages)
    for (int issued = 0; issued <= 5 * stages; ++issued) {
      const int stage = issued % stages;
      const uint32_t phase = static_cast<uint32_t>(issued / stages) & 1;
      for (uint32_t in_flight = 0; in_flight < (1u << stages); ++in_flight)
        for (int s = 0; s < stages; ++s) {
          const int loads = issued / stages + (s < stage);       // into stage s; a stage is filled again only when the last has landed
          const bool flying = loads > 0 && ((in_flight >> s) & 1);
#ifdef ITB_RING_ONE_PARITY
          const uint32_t parity = phase;                         // negative control: the same parity for all stages
#else
          const uint32_t parity = itb::ring_last_parity(s, itb::ring_position(stage, phase));
#endif
          ++checked;
          wrong += try_wait(loads - flying, parity) == flying;
        }
    }
  std::printf("ring model: %ld checked, %ld wrong\n", checked, wrong);
  return wrong != 0;
}
