// The rules by which a row's experts are ranked in FP32 and by which that ranking is too close to stand: the same in the router
// kernel, where a thread has the row (omni_router.cu), and in the routing of short batches, where a warp has it (route_kernel).
#pragma once
#include <stdint.h>

#include "omni_internal.h"

namespace {

// Unsigned integers in the order of the floats
__device__ __forceinline__ uint32_t ordered_key(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Logit and expert in one key: the larger logit first, among equal ones the lower expert.  The expert takes the place of
// the logit's last seven bits.
__device__ __forceinline__ uint32_t ranking_key(float logit, int expert) { return (ordered_key(logit) & ~127u) | (uint32_t)(127 - expert); }
__device__ __forceinline__ int ranked_expert(uint32_t key) { return 127 - (int)(key & 127u); }

// Whether the order of the first eight may be wrong, given the logits of the first nine: neighbours closer than twice the row's
// assumed accumulation error (it grows with the row's largest |logit|) and what the borrowed key bits can hide, 2^-14 of a logit
__device__ __forceinline__ bool near_tie(const float (&ranked)[9], float eps, float max_abs) {
    const float gap = 2.f * omni_row_eps(eps, max_abs) + fmaxf(fabsf(ranked[0]), fabsf(ranked[8])) * 6.1035156e-5f;
    bool close = false;
#pragma unroll
    for (int k = 0; k < 8; k++) close |= (ranked[k] - ranked[k + 1]) < gap;
    return close;
}

}  // namespace
