// Control flow of a CTA's K steps through a ring of shared-memory stages whose tensor-core work ends asynchronously. Kept
// apart from the kernel, and plain C++, so that the same code also runs under host threads (tests/test_mma_ring.py).
#pragma once

#ifdef __CUDACC__
#define ADOCK_RING_FN __device__ __forceinline__
#else
#define ADOCK_RING_FN inline
#endif

namespace adock {

// Called by all threads of the CTA:
//   wait(stage, parity)  waits, bounded, for the phase of that parity of the stage's barrier; false: gave up
//   fill(step, stage)    the thread's share of the stage's operands
//   any(flag)            CTA barrier; true in every thread if the flag is true in one
//   issue(step, stage)   one thread's tensor-core work on the stage, committed to the stage's barrier
// Returns (the same in every thread) whether all work has completed. Threads leave the loop together: whether a wait gave up
// is decided by the barrier's vote and not by a flag that a faster thread may already have set for the next step. Each
// issue's commit covers all work before it, so the wait for the last one that was issued, not the last step's, is the wait
// for everything in flight; it is tried twice (each bounded) before the caller goes on to free what that work uses.
template <int STAGES, typename WAIT, typename FILL, typename ANY, typename ISSUE>
ADOCK_RING_FN bool run_ring(int steps, const WAIT& wait, const FILL& fill, const ANY& any, const ISSUE& issue) {
    bool fail = false;
    int issued = 0;
    for (int it = 0; it < steps; ++it) {
        const int s = it % STAGES;
        const bool late = it >= STAGES && !wait(s, (unsigned)((it / STAGES - 1) & 1));
        if (!late) fill(it, s);   // else the stage may still be read
        fail = any(late);
        if (fail) break;
        issue(it, s);
        issued = it + 1;
    }
    bool late = false;
    if (issued > 0) {
        const int s = (issued - 1) % STAGES;
        const unsigned parity = (unsigned)(((issued - 1) / STAGES) & 1);
        late = !wait(s, parity) && !wait(s, parity);
    }
    return !any(fail || late);
}

}  // namespace adock
