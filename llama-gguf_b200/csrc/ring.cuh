// ring.cuh — the copies of a ring that may still be on their way.  Plain arithmetic (compiled by the host compiler in tests/test_rings_host.py).
#pragma once

#if defined(__CUDACC__)
#define RING_FN __host__ __device__ __forceinline__
#else
#define RING_FN inline
#endif

// A ring of N stages: copy t goes into stage t % N and completes phase t / N of that stage's barrier.  Copy t is asked for only after copy t - N has been
// consumed, so of the `asked` first copies the last N may be in flight.  wait(stage, parity) for each of them: what a loader that gives up does before its
// block may end -- a copy that lands after the shared memory has gone to another block would overwrite that block's.
template <int N, typename Wait> RING_FN void ring_in_flight(int asked, Wait wait) {
    for (int t = asked > N ? asked - N : 0; t < asked; t++) wait(t % N, (unsigned)(t / N) & 1u);
}
