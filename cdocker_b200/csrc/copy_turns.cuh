// copy_turns.cuh -- the turns of a CTA whose input comes by bulk copies into one buffer, the copies of one
// turn in flight at a time. Plain C++: the host test drives the same loop over a model of the barrier.
#pragma once

#ifdef __CUDACC__
#define CDK_TURNS __device__ __forceinline__
#else
#define CDK_TURNS inline
#endif

namespace cdk {

// Turns first, first + step, ... below end. The CTA's operations:
//   load(p)        arms the barrier's next phase and issues turn p's copies (one thread)
//   wait(parity)   bounded wait for the phase, sets the CTA's flag when it gives up
//   columns(p)     first half of the turn's work, ends with a CTA barrier
//   failed()       the flag
//   rows(p)        second half, ends with the fence and CTA barrier that free the buffer
//   drain(parity)  bounded wait for a phase whose copies may still be in flight
// Returns false when a wait gave up. Then no copy is issued after it (the phase is still armed: a second
// arrival would underflow its count, and the copies would share the buffer), and the one phase in flight
// has been drained: the buffer must not be used again, and the CTA may leave. Every thread takes the same way:
// the flag is set in wait only, which no thread enters again before all have read it behind the barrier of
// columns and passed that of rows.
template <class Cta>
CDK_TURNS bool copy_turns(int first, int step, int end, Cta& cta) {
  if (first < end) cta.load(first);
  unsigned int parity = 0;
#pragma unroll 1
  for (int p = first; p < end; p += step, parity ^= 1u) {
    cta.wait(parity);
    cta.columns(p);
    if (cta.failed()) {
      cta.drain(parity);
      return false;
    }
    cta.rows(p);
    if (p + step < end) cta.load(p + step);
  }
  return true;
}

}  // namespace cdk
