// How the four warps of an epilogue half, which share a barrier, agree once per work item whether to go on
// (omni_expert.cu).
// Plain C++ besides the barrier it is given, so that the order of its accesses is tested on the CPU.
#pragma once

#ifdef __CUDACC__
#define OMNI_MEET_FN __device__ __forceinline__
#else
#define OMNI_MEET_FN inline
#endif

// `ok`: this warp's waits for the item succeeded.  False for all warps as soon as it is false for one, so
// that they leave together and none is left in the barrier.  quit[2] starts as zeroes; items
// take its words in turn: behind the barrier a slow warp still reads the word of this item while a fast one may
// already report on the next, which is another word; the item after that lies behind a barrier
// that the slow warp has not reached yet.
template <class Word, class Barrier>
OMNI_MEET_FN bool warps_meet(Word *quit, int item, bool ok, Barrier barrier) {
    if (!ok) quit[item & 1] = 1;
    barrier();
    return quit[item & 1] == 0;
}
