/* Wait of a host thread for the number that the GPU writes after a launch's
 * results, in pinned host memory. */
#pragma once
#include <sched.h>
#include <stdint.h>

namespace gw {

/* The number of the next launch to wait for: never 0, which launches that
 * nobody waits for carry and leave in the slot. */
static inline uint32_t next_number(uint32_t n) { return n + 1u ? n + 1u : 1u; }

/* True once *slot holds seq.  busy(), asked now and then, says whether the
 * work that writes it is still under way; false: that work has ended (or
 * failed) and the number is not there. */
template <typename Busy>
static inline bool wait_number(const unsigned long long* slot, uint32_t seq, Busy busy) {
  for (;;) {
    for (int i = 0; i < 256; i++) {
      for (int k = 0; k < 64; k++)
        if (__atomic_load_n(slot, __ATOMIC_ACQUIRE) == seq) return true;
      sched_yield();
    }
    if (!busy()) return __atomic_load_n(slot, __ATOMIC_ACQUIRE) == seq;
  }
}

}  // namespace gw
