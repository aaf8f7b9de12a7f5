// How a CTA whose wait ran out gives the copies it has in flight a bounded chance to land before its shared memory
// goes to someone else (omni_expert.cu, omni_attn.cu).
// Plain C++ besides the barrier and the clock it is given, so that its bound is tested on the CPU.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define OMNI_LAND_FN __device__ __forceinline__
#else
#define OMNI_LAND_FN inline
#endif

constexpr uint64_t LAND_LIMIT_NS = 50000000ull, LAND_SETTLE_NS = 1000000ull;     // 50 ms, 1 ms

// armed[i]: parity of the phase in which copy i was announced last, -1 none.  landed(i, parity): that phase is complete.
// One limit over all of them: a barrier that two producers (or two CTAs) share does not complete once one of them has left, and says
// nothing then about the other's copies.  These land in microseconds; such a stage takes what is left of the limit, and those
// behind it are looked at once.  settle_ns is waited for in any case: the second CTA of a pair runs up to a ring ahead of the first, which announces
// the copies of both, and may have started copies into its own shared memory that the first has not announced when it gives up.
template <class Word, class Landed, class Clock>
OMNI_LAND_FN void copies_land(const Word *armed, int n, Landed landed, Clock now_ns, uint64_t limit_ns, uint64_t settle_ns) {
    const uint64_t t0 = now_ns();
    for (int i = 0; i < n; i++) {
        if (armed[i] < 0) continue;
        while (!landed(i, armed[i]) && now_ns() - t0 < limit_ns) {}
    }
    while (now_ns() - t0 < settle_ns) {}
}
