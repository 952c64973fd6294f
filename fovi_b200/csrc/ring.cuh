// Turns of the producer warps on a ring of shared-memory stages.  Plain C++ (the host test steps it against a model of the barriers).
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define FOVI_RING_FN __host__ __device__ __forceinline__
#else
#define FOVI_RING_FN inline
#endif

namespace fovi {

constexpr int PRODUCER_WARPS = 4;

// Stages 0, 1, 2, ... go to slots 0, 1, ..., nstage - 1 in turn; warp w fills stages w, w + step, w + 2 * step, ...  A slot is waited for by the
// parity of its "empty" barrier, which is unambiguous only while the waiter is at most one round ahead of the consumer.  A warp that was let into
// stage i - step knows that stage i - step - nstage has been consumed; the wait for stage i needs stage i - 2 * nstage consumed, so step may not
// exceed nstage: with four warps on three slots the wait returns at once and the copy lands on operands that the MMA has not read.  Warps beyond
// the ring's depth therefore stay idle.
struct RingTurn {
  uint32_t nstage, step, s, ph;   // s: this warp's slot, ph: parity of its "full" round (the "empty" wait is for ph ^ 1)
  bool idle;
  FOVI_RING_FN RingTurn(uint32_t warp, uint32_t nstage_)
      : nstage(nstage_), step(nstage_ < (uint32_t)PRODUCER_WARPS ? nstage_ : (uint32_t)PRODUCER_WARPS), s(warp), ph(0), idle(warp >= step) {}
  FOVI_RING_FN void next() {
    s += step;
    if (s >= nstage) { s -= nstage; ph ^= 1u; }   // step <= nstage: at most one round further
  }
};

}  // namespace fovi
