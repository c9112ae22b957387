/*
 * seg_state.h -- a state of the pointer jumping that finds the segments of a block of chain nodes
 * (chain.cu, k_seg_local), as a function of its own so that the rule is tested on the host.
 *
 * A state word holds the next state in its low STOP bits and the steps to it above; no steps: it
 * stops.  A block's path is shorter than 2^STOP steps.  A state on a cycle never stops, and the
 * jumping is in place, so that a round may add to a sum what the same round has made of another:
 * the steps stay at MOST once they get there, and a state that moves never reads as one that stops.
 */
#ifndef BRUNO_SEG_STATE_H_
#define BRUNO_SEG_STATE_H_

#include <cstdint>

#ifdef __CUDACC__
#define BRUNO_SEG_FN __host__ __device__ __forceinline__
#else
#define BRUNO_SEG_FN inline
#endif

namespace bruno_seg {

constexpr int STOP = 12;
constexpr uint32_t IDX = (1u << STOP) - 1, MOST = (1u << (32 - STOP)) - 1;

BRUNO_SEG_FN uint32_t steps(uint32_t w) { return w >> STOP; }

/* a state w that moves, on from its next state, which holds t and moves too */
BRUNO_SEG_FN uint32_t join(uint32_t w, uint32_t t) {
  const uint32_t s = steps(w) + steps(t);
  return (t & IDX) | ((s < MOST ? s : MOST) << STOP);
}

}  // namespace bruno_seg

#undef BRUNO_SEG_FN

#endif  // BRUNO_SEG_STATE_H_
