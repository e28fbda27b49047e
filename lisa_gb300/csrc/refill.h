// When a persistent traversal kernel takes new work: once this many of a
// warp's 32 lanes are idle.
#pragma once

#include <stdint.h>

namespace lisa {

// By default each kind of kernel has its own number, as its refill rounds
// differ in length.  Measured: closest hit 8 (4, 8, 10, 12, 16 tried: 14.05 ms
// a step of the 1.31 M-triangle icosphere box at 8, 14.19 at 12), emitter
// search 16 (12.1 ms against 12.4 at 12 and 12.7 at 8), whole paths 20
// (5.15 ms of 4 Mi Cornell box paths against 5.26 at 16 and 5.61 at 12).
constexpr uint32_t REFILL_TRACE = 8, REFILL_NEE = 16, REFILL_PATHS = 20;

// The option (1..32) is every kernel's, 0 the kernel's own.
constexpr uint32_t refill_idle_lanes(uint32_t option, uint32_t own) {
  return option == 0u ? own : option > 32u ? 32u : option;
}

}  // namespace lisa
