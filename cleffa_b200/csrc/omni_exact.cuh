// Device helpers shared by the routing kernels: warp-level top-k in the reference's order,
// the selection write-out, and exact logits (FP64 sums of exact BF16 products) with the
// re-evaluation of one near-tied router row by a group of eight warps.
//
// Reference behaviour (paths inside the reference project):
//   selection order / weights   metal/clef.metal:2347-2394  (omni_route)
//   exact logits                metal/clef.metal:2330-2345  (omni_router, compensated sum)
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "omni_internal.h"
#include "omni_select.cuh"

namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ float bf16_bits_to_float(uint32_t b16) { return __uint_as_float(b16 << 16); }

// ------------------------------------------------------------------ warp-level top-k
// Order: larger value first, equal values -> lower expert id first (clef.metal:2376-2382).
struct Best { double v; int id; };

__device__ __forceinline__ bool better(double v, int id, double ov, int oid) {
    return v > ov || (v == ov && id < oid);
}

__device__ __forceinline__ Best warp_argmax(double v, int id) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const double ov = __shfl_xor_sync(FULL, v, s);
        const int oid = __shfl_xor_sync(FULL, id, s);
        if (better(ov, oid, v, id)) { v = ov; id = oid; }
    }
    return Best{v, id};
}

// Each lane owns experts lane, lane+32, lane+64, lane+96.  Extracts the `n` best (n <= 9)
// in order into top_v/top_id (identical on every lane).  Taken entries become -inf.
template <int N>
__device__ __forceinline__ void warp_topn(double (&val)[4], int lane, double (&top_v)[N], int (&top_id)[N]) {
#pragma unroll
    for (int r = 0; r < N; r++) {
        double bv = val[0]; int bid = lane;
#pragma unroll
        for (int j = 1; j < 4; j++) if (better(val[j], lane + 32 * j, bv, bid)) { bv = val[j]; bid = lane + 32 * j; }
        const Best b = warp_argmax(bv, bid);
        top_v[r] = b.v; top_id[r] = b.id;
#pragma unroll
        for (int j = 0; j < 4; j++) if (lane + 32 * j == b.id) val[j] = -CUDART_INF;
    }
}

// The same order through integer keys and the warp-wide integer reductions, for the exact pass: a
// round of the shuffle search above costs about 300 clocks (five exchanges of a double and an id), one
// of these about 60.  Both searches of a row together: a block of 64 to 1030 tokens went from 218.6 to
// 216.7 us (64) and 239.6 to 238.2 (1030), two layers of 37 tokens from 451.7 to 448.2.
__device__ __forceinline__ float ordered_value(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }

// The 8th and 9th largest of the warp's 128 values (equal values count one by one).
__device__ __forceinline__ void warp_8th_9th(const float (&val)[4], int lane, float &v8, float &v9) {
    uint32_t k[4], top[9];
#pragma unroll
    for (int j = 0; j < 4; j++) k[j] = ordered_key(val[j]);
#pragma unroll
    for (int r = 0; r < 9; r++) {
        const uint32_t mine = max(max(k[0], k[1]), max(k[2], k[3]));
        top[r] = __reduce_max_sync(FULL, mine);
        const unsigned holders = __ballot_sync(FULL, mine == top[r]);
        if (lane == __ffs(holders) - 1) {
            bool taken = false;
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (!taken && k[j] == mine) { k[j] = 0; taken = true; }           // below the key of every number
        }
    }
    v8 = ordered_value(top[7]);
    v9 = ordered_value(top[8]);
}

// warp_topn<8> by keys: the high words decide, the low words and then the ids only among equals.
// Each reduction is a statement of its own: every lane has to take part, whatever its values are.
__device__ __forceinline__ void warp_top8(const double (&val)[4], int lane, double (&top_v)[9], int (&top_id)[9]) {
    uint64_t k[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint64_t u = (uint64_t)__double_as_longlong(val[j] + 0.0);           // -0 and +0 are equal
        k[j] = (u >> 63) ? ~u : (u | 0x8000000000000000ull);
    }
#pragma unroll
    for (int r = 0; r < 8; r++) {
        uint64_t bk = k[0];
        double bv = val[0];
        int bj = 0;
#pragma unroll
        for (int j = 1; j < 4; j++) if (k[j] > bk) { bk = k[j]; bv = val[j]; bj = j; }
        const uint32_t hi = (uint32_t)(bk >> 32), lo = (uint32_t)bk;
        const uint32_t top_hi = __reduce_max_sync(FULL, hi);
        bool best = hi == top_hi;
        unsigned m = __ballot_sync(FULL, best);
        if (m & (m - 1)) {                                                         // the same in all lanes
            const uint32_t top_lo = __reduce_max_sync(FULL, best ? lo : 0u);
            best = best && lo == top_lo;
            const uint32_t id = best ? (uint32_t)(lane + 32 * bj) : 0xffffffffu;
            const uint32_t first = __reduce_min_sync(FULL, id);
            m = __ballot_sync(FULL, best && id == first);
        }
        const int src = __ffs(m) - 1;
        top_v[r] = __shfl_sync(FULL, bv, src);
        top_id[r] = src + 32 * __shfl_sync(FULL, bj, src);
        if (lane == src) {
#pragma unroll
            for (int j = 0; j < 4; j++) if (j == bj) k[j] = 0;
        }
    }
}

// Lanes 0..7 hold the selected logits and ids in order; weights are softmax over the selected eight, which
// equals softmax over all experts renormalised by the selected sum (clef.metal:2393).
__device__ __forceinline__ void write_ranked(double v, int id, int lane, int32_t *ids, float *weights, long row) {
    const double first = __shfl_sync(FULL, v, 0);
    const double p = lane < 8 ? exp(v - first) : 0.0;
    double sum = p;
#pragma unroll
    for (int s = 4; s > 0; s >>= 1) sum += __shfl_xor_sync(FULL, sum, s);
    if (lane < 8) { ids[row * 8 + lane] = id; weights[row * 8 + lane] = (float)(p / sum); }
}
__device__ __forceinline__ void write_selection(const double (&top_v)[9], const int (&top_id)[9], int lane,
                                                int32_t *ids, float *weights, long row) {
    double v = 0.0;
    int id = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) if (lane == k) { v = top_v[k]; id = top_id[k]; }
    write_ranked(v, id, lane, ids, weights, row);
}

__device__ __forceinline__ void write_fallback(int lane, int32_t *ids, float *weights, long row, uint32_t *status) {
    // clef.metal:2362-2367: report once, keep the pass well-defined.
    if (lane == 0) atomicOr(status, OMNI_ST_NONFINITE);
    if (lane < 8) { ids[row * 8 + lane] = lane; weights[row * 8 + lane] = 0.0f; }
}

// ------------------------------------------------------------------ exact dot (FP64 sum of exact products)
// A lane owns K elements lane*8 + 256*i .. +7 (i < 8): one 16-byte load per step.
struct XRow { uint4 q[8]; };

__device__ __forceinline__ XRow load_xrow(const __nv_bfloat16 *xn, long row, int lane) {
    XRow r;
    const uint4 *p = reinterpret_cast<const uint4 *>(xn + row * OMNI_H);
#pragma unroll
    for (int i = 0; i < 8; i++) r.q[i] = __ldg(p + lane + 32 * i);
    return r;
}

// bf16*bf16 is exact in FP32 (8+8 significand bits); the FP64 sum of 2048 such terms is
// accurate to ~1e-13, far inside the 1e-9 bound of tests/test_omni_router.m:44.
__device__ __forceinline__ double exact_dot(const XRow &x, const __nv_bfloat16 *wrow, int lane) {
    const uint4 *p = reinterpret_cast<const uint4 *>(wrow);
    uint4 w[8];
#pragma unroll
    for (int i = 0; i < 8; i++) w[i] = __ldg(p + lane + 32 * i);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};      // four chains: the FP64 adds overlap instead of serialising
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t xu[4] = {x.q[i].x, x.q[i].y, x.q[i].z, x.q[i].w};
        const uint32_t wu[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            acc[j] += (double)(bf16_bits_to_float(xu[j] & 0xffffu) * bf16_bits_to_float(wu[j] & 0xffffu));
            acc[j] += (double)(bf16_bits_to_float(xu[j] >> 16) * bf16_bits_to_float(wu[j] >> 16));
        }
    }
    double sum = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(FULL, sum, s);
    return sum;
}

// The same sum for the exact pass, by eight warps and for EXACT_BATCH experts at once.  A lane owns eight of
// the 2048 K elements (its warp's 256), so the weights of all candidates of a row -- nine or ten as a
// rule -- are in flight together; with a warp per candidate a row took three rounds of loads and sums one after
// the other.  A BF16 weight becomes a double by moving its bits: sign and exponent field in the
// upper word of a double stand for the value times 2^-896, denormals included, and the sum is scaled back
// exactly (the conversion instruction runs at a quarter of the rate of the FP64 adds).  Nonfinite weights
// do not come here: the logits of their rows are nonfinite.
constexpr int EXACT_BATCH = 12, EXACT_WARPS = 8, EXACT_THREADS = 32 * EXACT_WARPS;
__device__ __forceinline__ double bf16_lo_scaled(uint32_t u) {
    return __hiloint2double((int)(((u << 16) & 0x80000000u) | ((u & 0x7fffu) << 13)), 0);
}
__device__ __forceinline__ double bf16_hi_scaled(uint32_t u) {
    return __hiloint2double((int)((u & 0x80000000u) | ((u >> 3) & 0x0fffe000u)), 0);
}
constexpr double EXACT_UNSCALE = 0x1p896;

struct ExactScratch {
    double part[EXACT_WARPS][EXACT_BATCH];
    double exact[OMNI_E];                  // by expert; -inf where nothing was evaluated
    double sorted_v[8];
    int sorted_id[8];
    float approx[OMNI_E];                  // by candidate
    int cand[OMNI_E];                      // expert of each candidate
    int n;                                 // candidates
    double bound;                          // the row's error bound
};

// One warp lists the candidates of a row: every expert that can still reach the top eight (approximate
// logit within twice the row's error bound of the approximate 8th) and the approximate 9th.
__device__ __forceinline__ void recheck_list(const float (&approx)[4], float eps, int lane, ExactScratch &sc) {
    float max_abs = 0.f;
#pragma unroll
    for (int j = 0; j < 4; j++) max_abs = fmaxf(max_abs, fabsf(approx[j]));
    max_abs = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(max_abs)));          // not negative: ordered like its bits
    const double bound = (double)omni_row_eps(eps, max_abs);
    float v8, v9;
    warp_8th_9th(approx, lane, v8, v9);
    const double floor_v = fmin((double)v8 - 2.0 * bound, (double)v9);
    int n = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const bool in = (double)approx[j] >= floor_v;
        const unsigned m = __ballot_sync(FULL, in);
        const int at = n + __popc(m & ((1u << lane) - 1u));
        if (in) { sc.cand[at] = lane + 32 * j; sc.approx[at] = approx[j]; }
        sc.exact[lane + 32 * j] = -CUDART_INF;
        n += __popc(m);
    }
    if (lane == 0) { sc.n = n; sc.bound = bound; }
}

// Re-evaluates one flagged row with eight warps (256 threads): exact logits of the candidates that recheck_list has
// left in the scratch (behind a barrier), then the final order by warp 0.  `xq`: this lane's part of the row
// (recheck_x).  `sync` is a barrier over exactly these threads.  With `segcount` given (expert counts per 256-assignment
// segment, taken from the ids being replaced), the counts follow the ids that change.
//
// What the pass learns is written back: every logit it evaluated is replaced by its exact value
// as a float pair (hi into `logits`, the remainder into `low` when given), so that a capture of
// the row shows logits that agree with the ids chosen from them (clef_metal_omni.m:118-130
// prints hi+lo).  And the assumed error bound is checked on the way: an approximate logit
// further than the bound from its exact value raises OMNI_ST_ROUTER_EPS.
__device__ __forceinline__ int recheck_k(int lane, int warp) { return warp * (OMNI_H / EXACT_WARPS) + lane * 8; }
__device__ __forceinline__ uint4 recheck_x(const __nv_bfloat16 *xn, long row, int lane, int warp) {
    return __ldg(reinterpret_cast<const uint4 *>(xn + row * OMNI_H + recheck_k(lane, warp)));
}

template <typename Sync>
__device__ __forceinline__ void recheck_row(const uint4 &xq, const __nv_bfloat16 *__restrict__ w,
                                            const float *__restrict__ bias, float *__restrict__ logits,
                                            float *__restrict__ low, long row, int32_t *__restrict__ ids,
                                            float *__restrict__ weights, int32_t *__restrict__ segcount,
                                            uint32_t *__restrict__ status, ExactScratch &sc, int lane, int warp, Sync sync) {
    const int koff = recheck_k(lane, warp), n = sc.n;
    const int old_id = segcount && warp == 0 && lane < 8 ? ids[row * 8 + lane] : 0;
    double x[8];
    {
        const uint32_t u[4] = {xq.x, xq.y, xq.z, xq.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            x[2 * j] = (double)bf16_bits_to_float(u[j] & 0xffffu);
            x[2 * j + 1] = (double)bf16_bits_to_float(u[j] >> 16);
        }
    }
    double mine_v = 0.0;                                  // warp 0: candidate `lane` of a row with at most EXACT_BATCH of them
    for (int b0 = 0; b0 < n; b0 += EXACT_BATCH) {
        uint4 wq[EXACT_BATCH];
#pragma unroll
        for (int i = 0; i < EXACT_BATCH; i++)
            wq[i] = b0 + i < n ? __ldg(reinterpret_cast<const uint4 *>(w + (long)sc.cand[b0 + i] * OMNI_H + koff)) : make_uint4(0, 0, 0, 0);
        double s[EXACT_BATCH];
#pragma unroll
        for (int i = 0; i < EXACT_BATCH; i++) {
            const uint32_t u[4] = {wq[i].x, wq[i].y, wq[i].z, wq[i].w};
            s[i] = 0.0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                s[i] = fma(x[2 * j], bf16_lo_scaled(u[j]), s[i]);
                s[i] = fma(x[2 * j + 1], bf16_hi_scaled(u[j]), s[i]);
            }
        }
        // sums over the warp's lanes, four candidates at a time: lanes with bit 4 (then bit 3) set keep the
        // upper half of the values and hand over the lower one, so four sums take six exchanges and not twenty
#pragma unroll
        for (int q = 0; q < EXACT_BATCH; q += 4) {
            const bool h16 = lane & 16, h8 = lane & 8;
            double a0 = h16 ? s[q + 2] : s[q], a1 = h16 ? s[q + 3] : s[q + 1];
            const double g0 = h16 ? s[q] : s[q + 2], g1 = h16 ? s[q + 1] : s[q + 3];
            a0 += __shfl_xor_sync(FULL, g0, 16);
            a1 += __shfl_xor_sync(FULL, g1, 16);
            double r = h8 ? a1 : a0;
            r += __shfl_xor_sync(FULL, h8 ? a0 : a1, 8);
#pragma unroll
            for (int d = 4; d > 0; d >>= 1) r += __shfl_xor_sync(FULL, r, d);
            if ((lane & 7) == 0) sc.part[warp][q + (lane >> 3)] = r;      // lane 8k holds candidate q + k
        }
        sync();
        if (warp == 0 && lane < EXACT_BATCH && b0 + lane < n) {
            double v = 0.0;
#pragma unroll
            for (int k = 0; k < EXACT_WARPS; k++) v += sc.part[k][lane];
            v *= EXACT_UNSCALE;
            const int e = sc.cand[b0 + lane];
            if (bias) v += (double)bias[e];
            if (fabs(v - (double)sc.approx[b0 + lane]) > sc.bound) atomicOr(status, OMNI_ST_ROUTER_EPS);
            const float hi = (float)v;
            logits[row * OMNI_E + e] = hi;
            if (low) low[row * OMNI_E + e] = (float)(v - (double)hi);
            sc.exact[e] = mine_v = v;
        }
        if (b0 + EXACT_BATCH < n) sync();                 // the partial sums are read before the next batch's are written
    }
    if (warp == 0) {
        __syncwarp();
        double v = -CUDART_INF;
        int id = 0;
        if (n <= EXACT_BATCH) {
            // order of a few candidates: each counts those in front of it
            const int e = lane < n ? sc.cand[lane] : OMNI_E;
            int rank = lane < n ? 0 : 32;
            for (int j = 0; j < n; j++) {
                const double ov = __shfl_sync(FULL, mine_v, j);
                const int oid = __shfl_sync(FULL, e, j);
                if (j != lane && better(ov, oid, mine_v, e)) rank++;
            }
            if (rank < 8) { sc.sorted_v[rank] = mine_v; sc.sorted_id[rank] = e; }
            __syncwarp();
            if (lane < 8) { v = sc.sorted_v[lane]; id = sc.sorted_id[lane]; }
        } else {
            double exact[4], fin_v[9];
            int fin_id[9];
#pragma unroll
            for (int j = 0; j < 4; j++) exact[j] = sc.exact[lane + 32 * j];
            warp_top8(exact, lane, fin_v, fin_id);
#pragma unroll
            for (int k = 0; k < 8; k++) if (lane == k) { v = fin_v[k]; id = fin_id[k]; }
        }
        write_ranked(v, id, lane, ids, weights, row);
        if (segcount && lane < 8 && id != old_id) {       // a row's eight assignments share one segment
            int32_t *c = segcount + (row * OMNI_TOP / OMNI_SEG) * OMNI_E;
            atomicSub(c + old_id, 1);
            atomicAdd(c + id, 1);
        }
    }
}

}  // namespace
