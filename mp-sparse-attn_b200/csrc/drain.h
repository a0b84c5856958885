// What the producers of a pair of CTAs still have to wait for when one or both leave a ring of stages early (csrc/gemm.cu).
// Every stage's copies, of both CTAs, report to one barrier of the first CTA, which the first CTA arms with the bytes of both.  A CTA
// that stopped earlier than the other leaves stages behind that only one of the two has filled: they never complete by themselves.
// Plain functions of numbers, so that the host can check them against a model of the barriers.
#pragma once

#ifdef __CUDACC__
#define MPSA_HD __host__ __device__ __forceinline__
#else
#define MPSA_HD inline
#endif

namespace mpsa {

// Stages are counted from 0 over the whole run; n0, n1: stages that the first and the second CTA have requested copies for;
// `ring`: stages of the ring.  A stage is requested only once the one `ring` before it has been used, so only the last `ring` of the
// larger count can have copies in flight, and the counts differ by `ring` at most.
MPSA_HD int drain_first(int n0, int n1, int ring) {
  const int n = n0 > n1 ? n0 : n1;
  return n > ring ? n - ring : 0;
}
MPSA_HD int drain_end(int n0, int n1) { return n0 > n1 ? n0 : n1; }

// What the first CTA does to the barrier of stage u before it waits for that phase.
enum DrainStep {
  DRAIN_WAIT = 0,      // both CTAs' copies are on their way and the phase is armed for them
  DRAIN_ARM = 1,       // only the second CTA's: arm the phase with one CTA's bytes
  DRAIN_FILL = 2,      // armed for both, only the first CTA's came: count the other's bytes off
};
MPSA_HD DrainStep drain_step(int u, int n0, int n1) { return u >= n0 ? DRAIN_ARM : u >= n1 ? DRAIN_FILL : DRAIN_WAIT; }

}  // namespace mpsa
