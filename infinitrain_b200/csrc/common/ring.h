// The ring of stages that a producer fills with asynchronous loads, one mbarrier a stage.  Host and device.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define ITB_HOST_DEVICE __host__ __device__
#else
#define ITB_HOST_DEVICE
#endif

namespace itb {

// Where a producer stopped: the stage that it would have filled next, in a lap of parity `phase` (the first lap: 0).
ITB_HOST_DEVICE constexpr uint32_t ring_position(int stage, uint32_t phase) {
  return (static_cast<uint32_t>(stage) << 1) | (phase & 1);
}

// The parity to wait for at stage `s` until the last load that went into it has landed.  Stages before the position were
// filled in its lap, the others in the lap before; in the first lap those were not filled at all, and the wait for the phase
// before a barrier's first returns at once.
ITB_HOST_DEVICE constexpr uint32_t ring_last_parity(int s, uint32_t position) {
  return s < static_cast<int>(position >> 1) ? (position & 1) : (position & 1) ^ 1;
}

}  // namespace itb
