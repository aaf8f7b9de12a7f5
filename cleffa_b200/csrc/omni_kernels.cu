// HBM- and latency-bound stages of the Clef-Omni MoE block for sm_100a: exact re-evaluation of
// near-tied router rows, deterministic stable counting sort, weighted combine, the RMSNorm in
// front of the block, plus what the default path only uses for checks or caller-supplied
// routing: warp-level top-k selection, the stand-alone histogram, the row gather and plain
// CUDA-core kernels for the two expert products.  The tensor-core kernels live in omni_expert.cu,
// omni_router.cu and omni_attn.cu.
//
// Reference behaviour these kernels reproduce (paths inside the reference project):
//   selection / weights     metal/clef.metal:2347-2394  (omni_route)
//   exact logits            metal/clef.metal:2330-2345  (omni_router, compensated sum)
//   histogram / sort        metal/clef.metal:2396-2443  (omni_assign_count/offsets/scatter)
//   gather                  metal/clef.metal:2445-2453  (omni_gather)
//   combine                 metal/clef.metal:2494-2523  (omni_combine)
//   route capture           metal/clef.metal:2526-2539  (omni_trace)
//   norm before the block   metal/clef.metal:190-204    (rmsnorm_f32)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "omni_internal.h"
#include "omni_exact.cuh"
#include "omni_pdl.cuh"

namespace {

// ------------------------------------------------------------------ check-path logits
// One block per token, one thread per expert; FP32 accumulation.  Slow: a cross-check for
// the tensor-core router, never the default.
__global__ void __launch_bounds__(128) router_simple_kernel(const __nv_bfloat16 *__restrict__ xn,
                                                            const __nv_bfloat16 *__restrict__ w,
                                                            const float *__restrict__ bias, float *__restrict__ logits) {
    __shared__ float xs[OMNI_H];
    const long t = blockIdx.x;
    for (int k = threadIdx.x; k < OMNI_H; k += 128) xs[k] = __bfloat162float(xn[t * OMNI_H + k]);
    __syncthreads();
    const int e = threadIdx.x;
    const uint4 *wr = reinterpret_cast<const uint4 *>(w + (long)e * OMNI_H);
    float acc = 0.f;
    for (int k8 = 0; k8 < OMNI_H / 8; k8++) {
        const uint4 q = __ldg(wr + k8);
        const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            acc = fmaf(xs[k8 * 8 + 2 * j], bf16_bits_to_float(u[j] & 0xffffu), acc);
            acc = fmaf(xs[k8 * 8 + 2 * j + 1], bf16_bits_to_float(u[j] >> 16), acc);
        }
    }
    logits[t * OMNI_E + e] = acc + (bias ? bias[e] : 0.f);
}

// ------------------------------------------------------------------ selection from stored logits
// One warp per token.  Rows whose ranked logits are closer than 2*eps anywhere in the first
// nine (or every row when exact_all) are appended to flag_rows for the exact pass; eps is the
// row's error bound (omni_row_eps).
__global__ void __launch_bounds__(256) select_kernel(const float *__restrict__ logits, int T, float eps, int exact_all,
                                                     int32_t *__restrict__ ids, float *__restrict__ weights,
                                                     int32_t *__restrict__ flag_rows, int32_t *__restrict__ n_flag,
                                                     uint32_t *__restrict__ status) {
    const int lane = threadIdx.x & 31;
    const long row = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= T) return;
    double val[4];
    bool bad = false;
    float max_abs = 0.f;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float f = logits[row * OMNI_E + lane + 32 * j];
        bad |= !isfinite(f);
        val[j] = (double)f;
        max_abs = fmaxf(max_abs, fabsf(f));
    }
    if (__any_sync(FULL, bad)) { write_fallback(lane, ids, weights, row, status); return; }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) max_abs = fmaxf(max_abs, __shfl_xor_sync(FULL, max_abs, s));
    const double bound = (double)omni_row_eps(eps, max_abs);
    double top_v[9]; int top_id[9];
    warp_topn<9>(val, lane, top_v, top_id);
    bool close = exact_all != 0;
#pragma unroll
    for (int k = 0; k < 8; k++) close |= (top_v[k] - top_v[k + 1]) < 2.0 * bound;
    write_selection(top_v, top_id, lane, ids, weights, row);
    if (close && lane == 0) { const int at = atomicAdd(n_flag, 1); if (at < OMNI_CHUNK) flag_rows[at] = (int32_t)row; }
}

// This block's share of a request for memory to be brought into L2, spread over the grid.
__device__ __forceinline__ void prefetch_share(const char *p, int pieces) {
    for (int i = blockIdx.x + gridDim.x * threadIdx.x; i < pieces; i += gridDim.x * blockDim.x)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p + (size_t)i * OMNI_PREFETCH_PIECE), "r"(OMNI_PREFETCH_PIECE) : "memory");
}

// One block per flagged row.  Its blocks become resident while the router runs, when device
// memory is idle: with `prefetch` given they ask for that much of the expert weights to be
// brought into L2 meanwhile.  That takes blocks on every SM: 48 MiB requested by the 37 blocks of a norm
// kernel held that kernel up by 29 us.
template <bool PREFETCH>
__global__ void __launch_bounds__(EXACT_THREADS) recheck_kernel(const __nv_bfloat16 *__restrict__ xn,
                                                      const __nv_bfloat16 *__restrict__ w,
                                                      const float *__restrict__ bias, float *__restrict__ logits,
                                                      float *__restrict__ low, const int32_t *__restrict__ flag_rows,
                                                      const int32_t *__restrict__ n_flag, int T, float eps,
                                                      int32_t *__restrict__ ids, float *__restrict__ weights,
                                                      int32_t *__restrict__ segcount, uint32_t *__restrict__ status,
                                                      const char *prefetch, int prefetch_pieces) {
    __shared__ ExactScratch scratch;
    if (PREFETCH) prefetch_share(prefetch, prefetch_pieces);
    dep_wait();
    dep_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int n = *n_flag;
    if (n > T) n = T;                  // a count left by a pass that failed half-way can be no larger than this
    for (int f = blockIdx.x; f < n; f += gridDim.x) {
        const long row = flag_rows[f];
        const uint4 xq = recheck_x(xn, row, lane, warp);
        __syncthreads();                                   // the row before is done with the scratch
        if (warp == 0) {
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = logits[row * OMNI_E + lane + 32 * j];
            recheck_list(v, eps, lane, scratch);
        }
        __syncthreads();
        recheck_row(xq, w, bias, logits, low, row, ids, weights, segcount, status, scratch, lane, warp, [] { __syncthreads(); });
    }
}

// Exact logits for every (token, expert): tests only (tests/test_omni_router.m).
__global__ void __launch_bounds__(128) router_exact_kernel(const __nv_bfloat16 *__restrict__ xn,
                                                           const __nv_bfloat16 *__restrict__ w,
                                                           const float *__restrict__ bias, double *__restrict__ out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long row = blockIdx.x;
    const XRow x = load_xrow(xn, row, lane);
    for (int e = warp; e < OMNI_E; e += 4) {
        double v = exact_dot(x, w + (long)e * OMNI_H, lane);
        if (bias) v += (double)bias[e];
        if (lane == 0) out[row * OMNI_E + e] = v;
    }
}

// omni_route on caller-supplied hi/lo pairs (tests/test_omni_moe.m modes).
__global__ void __launch_bounds__(256) route_pairs_kernel(const float *__restrict__ hi, const float *__restrict__ lo,
                                                          int rows, int32_t *__restrict__ ids,
                                                          float *__restrict__ weights, uint32_t *__restrict__ status) {
    const int lane = threadIdx.x & 31;
    const long row = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    double val[4];
    bool bad = false;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float h = hi[row * OMNI_E + lane + 32 * j];
        const float l = lo ? lo[row * OMNI_E + lane + 32 * j] : 0.f;
        bad |= !isfinite(h) || !isfinite(l);
        val[j] = (double)h + (double)l;
    }
    if (__any_sync(FULL, bad)) { write_fallback(lane, ids, weights, row, status); return; }
    double top_v[9]; int top_id[9];
    warp_topn<9>(val, lane, top_v, top_id);
    write_selection(top_v, top_id, lane, ids, weights, row);
}

// ------------------------------------------------------------------ histogram + stable counting sort
// Assignment i = t*8 + k (k = rank in the descending top-8).  A segment is 256 consecutive
// assignments handled by one warp; segment histograms make the sort parallel while the
// result stays the serial, stable bucket order of clef.metal:2418-2443.
__global__ void __launch_bounds__(256) assign_hist_kernel(const int32_t *__restrict__ ids, int A, int nseg,
                                                          int32_t *__restrict__ segcount, uint32_t *__restrict__ status) {
    __shared__ int hist[8][OMNI_E];
    dep_wait();
    dep_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int seg = blockIdx.x * 8 + warp;
#pragma unroll
    for (int j = 0; j < 4; j++) hist[warp][lane + 32 * j] = 0;
    __syncwarp();
    if (seg < nseg) {
        for (int it = 0; it < OMNI_SEG / 32; it++) {
            const int i = seg * OMNI_SEG + it * 32 + lane;
            int e = i < A ? ids[i] : -1;
            if (i < A && (e < 0 || e >= OMNI_E)) { atomicOr(status, OMNI_ST_BAD_ID); e &= OMNI_E - 1; }
            const unsigned m = __match_any_sync(FULL, e);
            if (e >= 0 && lane == __ffs(m) - 1) hist[warp][e] += __popc(m);
            __syncwarp();
        }
#pragma unroll
        for (int j = 0; j < 4; j++) segcount[(long)seg * OMNI_E + lane + 32 * j] = hist[warp][lane + 32 * j];
    }
}

// Scan over the experts, shared by the two kernels that place assignments; called by all 256 threads of a
// block with the number of rows of expert tid % 128.  Returns the expert's offset to the first 128 threads. With
// `publish` the other 128 also write counts, offsets and the token-tile list of the expert products and reset the
// counters that the rest of the pass starts from: off the path of the threads that go on to place assignments
// (3600 clocks while those did it themselves).
struct ExpertScan { int warp_rows[4], warp_tiles[4]; int4 key[OMNI_E / 4], cnt[OMNI_E / 4]; };

__device__ __forceinline__ int scan_experts(ExpertScan &sm, int total, const omni_sort_state &st, bool publish) {
    const int e = threadIdx.x & (OMNI_E - 1), lane = threadIdx.x & 31;
    const bool publisher = threadIdx.x >= OMNI_E;
    // the router and the exact pass of this chunk are done with the flagged-row count: keep it
    // for introspection and clear it for the next router launch (no memset between passes)
    const int flagged = publisher && publish && e == 0 && st.n_flag ? st.n_flag[0] : 0;
    // inclusive scans over the 128 experts (rows and token tiles): shuffles inside each of
    // four warps (both halves of the block hold the same numbers), then the totals of the warps before
    const int nt = (total + st.tile_n - 1) / st.tile_n;
    int rows_incl = total, tiles_incl = nt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int a = __shfl_up_sync(FULL, rows_incl, d), b = __shfl_up_sync(FULL, tiles_incl, d);
        if (lane >= d) { rows_incl += a; tiles_incl += b; }
    }
    // order of the tile list: falling tile length, equal ones by expert
    int key = 0;
    if (!publisher) {
        if (lane == 31) sm.warp_rows[e >> 5] = rows_incl;
    } else {
        key = (nt ? total / nt * OMNI_E : 0) + OMNI_E - 1 - e;
        if (lane == 31) sm.warp_tiles[e >> 5] = tiles_incl;
        reinterpret_cast<int *>(sm.key)[e] = key;
        reinterpret_cast<int *>(sm.cnt)[e] = nt;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 3; q++) if (q < (e >> 5)) { rows_incl += sm.warp_rows[q]; tiles_incl += sm.warp_tiles[q]; }
    const int off = rows_incl - total;
    if (!publisher || !publish) return off;
    st.counts[e] = total;
    st.offsets[e] = off;
    if (e == OMNI_E - 1) st.offsets[OMNI_E] = rows_incl;
    // Expert-major tile list, the experts in order of falling tile length (ties by id): the work
    // items of the persistent expert kernels are claimed in list order, so the longest come first
    // and the short ones fill the end of the launch.  Rows and offsets stay in expert order.  Both products
    // read this list: with one in expert order for the down product a block took 437.5 us against 438 (4096
    // tokens), 742 against 743 (8192), 1367 against 1374 (16384), 653 against 655 (8192, skewed).
    int first = tiles_incl - nt;
    if (st.longest_first) {
        first = 0;
#pragma unroll 8
        for (int o = 0; o < OMNI_E / 4; o++) {
            const int4 k = sm.key[o], c = sm.cnt[o];
            first += (k.x > key ? c.x : 0) + (k.y > key ? c.y : 0) + (k.z > key ? c.z : 0) + (k.w > key ? c.w : 0);
        }
    }
    // an expert's rows are split into nt tiles of near-equal length: tiles that share a
    // weight tile then advance at the same pace and meet in L2
    const int base = nt ? total / nt : 0, extra = nt ? total % nt : 0;
    for (int j = 0; j < nt; j++)
        st.ttiles[first + j] = omni_ttile{e, off + j * base + min(j, extra), base + (j < extra), first | (nt << 16)};
    if (e < 8) st.sched[e] = 0;
    if (e == OMNI_E - 1) *st.n_ttiles = tiles_incl;
    if (e == 0 && st.n_flag) { st.n_flag[1] = flagged; st.n_flag[0] = 0; }
    return off;
}

// Counting sort behind the segment histograms: every block takes eight segments (a warp each) and works
// out for itself where they start, from all of the histograms -- 512 bytes per segment from L2,
// 256 KiB at 16384 tokens.  As a kernel of one block in front of the scatter that scan was a link
// of its own in the chain of launches, and its single block took 15 us at 16384 tokens.
constexpr int ASSIGN_SEGS = 8, ASSIGN_THREADS = 32 * ASSIGN_SEGS;
static_assert(ASSIGN_THREADS == 2 * OMNI_E && EXACT_THREADS == 2 * OMNI_E, "scan_experts: half of the threads publish");
__global__ void __launch_bounds__(ASSIGN_THREADS) assign_kernel(const int32_t *__restrict__ ids, int A, int nseg, omni_sort_state st) {
    __shared__ ExpertScan scan;
    __shared__ int4 all[ASSIGN_SEGS][OMNI_E / 4], front[ASSIGN_SEGS][OMNI_E / 4];     // sums of a warp's share of the segments
    __shared__ int4 own[ASSIGN_SEGS][OMNI_E / 4];                                     // counts of this block's segments, then where they start
    __shared__ unsigned mask[ASSIGN_SEGS][OMNI_E];
    dep_wait();
    dep_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, e = threadIdx.x & (OMNI_E - 1);
    const int seg0 = blockIdx.x * ASSIGN_SEGS, seg = seg0 + warp;
    const int t = seg * 32 + lane;                                                    // a segment is the 8 assignments of 32 tokens
    const bool have = t * OMNI_TOP < A;
    int id[OMNI_TOP];                                                                 // loaded while the histograms are summed
    if (have && !((uintptr_t)ids & 15)) {
        const int4 a = *(reinterpret_cast<const int4 *>(ids) + 2 * t), b = *(reinterpret_cast<const int4 *>(ids) + 2 * t + 1);
        id[0] = a.x; id[1] = a.y; id[2] = a.z; id[3] = a.w; id[4] = b.x; id[5] = b.y; id[6] = b.z; id[7] = b.w;
    } else {
#pragma unroll
        for (int k = 0; k < OMNI_TOP; k++) id[k] = have ? ids[t * OMNI_TOP + k] : 0;
    }
#pragma unroll
    for (int k = 0; k < OMNI_TOP; k++) id[k] &= OMNI_E - 1;
    const int4 *hist = reinterpret_cast<const int4 *>(st.segcount) + lane;
    auto add = [](int4 &a, const int4 &b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; };
    int4 mine = seg < nseg ? hist[(long)seg * (OMNI_E / 4)] : make_int4(0, 0, 0, 0), fr = make_int4(0, 0, 0, 0);
    own[warp][lane] = mine;
#pragma unroll 8
    for (int s = warp; s < seg0; s += ASSIGN_SEGS) add(fr, hist[(long)s * (OMNI_E / 4)]);
    add(mine, fr);
#pragma unroll 8
    for (int s = seg + ASSIGN_SEGS; s < nseg; s += ASSIGN_SEGS) add(mine, hist[(long)s * (OMNI_E / 4)]);
    all[warp][lane] = mine;
    front[warp][lane] = fr;
#pragma unroll
    for (int j = 0; j < 4; j++) mask[warp][lane + 32 * j] = 0;
    __syncthreads();
    // a token's experts are distinct as a rule, so the tokens of a segment that chose an expert are a mask of
    // 32 bits and a token's rank among them a count of bits
    bool twice = false;
    if (have)
#pragma unroll
        for (int k = 0; k < OMNI_TOP; k++) twice |= (atomicOr(&mask[warp][id[k]], 1u << lane) >> lane) & 1;
    int total = 0, run = 0;
#pragma unroll
    for (int q = 0; q < ASSIGN_SEGS; q++) {
        total += reinterpret_cast<const int *>(all[q])[e];
        run += reinterpret_cast<const int *>(front[q])[e];
    }
    run += scan_experts(scan, total, st, blockIdx.x == 0);
    if (threadIdx.x < OMNI_E)
#pragma unroll
        for (int q = 0; q < ASSIGN_SEGS; q++) {
            int *c = reinterpret_cast<int *>(own[q]) + e;
            const int n = *c;
            *c = run;
            run += n;
        }
    __syncthreads();
    if (seg >= nseg) return;
    int *base = reinterpret_cast<int *>(own[warp]);
    const unsigned lt = (1u << lane) - 1u;
    if (!__any_sync(FULL, twice)) {
        if (!have) return;
        int row[OMNI_TOP];
#pragma unroll
        for (int k = 0; k < OMNI_TOP; k++) {
            row[k] = base[id[k]] + __popc(mask[warp][id[k]] & lt);
            st.rowmap[row[k]] = t;
        }
        if (!((uintptr_t)st.slots & 15)) {
            reinterpret_cast<int4 *>(st.slots)[2 * t] = make_int4(row[0], row[1], row[2], row[3]);
            reinterpret_cast<int4 *>(st.slots)[2 * t + 1] = make_int4(row[4], row[5], row[6], row[7]);
        } else {
#pragma unroll
            for (int k = 0; k < OMNI_TOP; k++) st.slots[t * OMNI_TOP + k] = row[k];
        }
        return;
    }
    // caller-supplied ids that name an expert twice for one token: assignments in order, 32 at a time
    for (int it = 0; it < OMNI_SEG / 32; it++) {
        const int i = seg * OMNI_SEG + it * 32 + lane;
        const int ei = i < A ? (ids[i] & (OMNI_E - 1)) : -1;
        const unsigned m = __match_any_sync(FULL, ei);
        if (ei >= 0) {
            const int row = base[ei] + __popc(m & lt);
            st.slots[i] = row;
            st.rowmap[row] = i >> 3;
        }
        __syncwarp();
        if (ei >= 0 && lane == __ffs(m) - 1) base[ei] += __popc(m);
        __syncwarp();
    }
}

// ------------------------------------------------------------------ routing of short batches
// Behind router_part_kernel: selection, exact pass and counting sort of up to ROUTE_MAX_ROWS tokens in one
// launch.  A block per token: its first warp ranks the logits and forms the weights -- the rules and, in
// rank order, the sums of the router kernel's own selection, bit for bit -- and all eight warps re-decide
// the row when it is too close.  The last block to finish sorts the assignments of the whole batch.  In separate
// launches (selection in the router, exact pass, scan, scatter) each of these steps takes 1 to 3 us and
// the way from one to the next as much again.
constexpr int ROUTE_SEGS = OMNI_ROUTE_MAX_ROWS / 32;
template <bool PREFETCH>
__global__ void __launch_bounds__(EXACT_THREADS) route_kernel(const __nv_bfloat16 *__restrict__ xn, const __nv_bfloat16 *__restrict__ w,
                                                              const float *__restrict__ bias, float *__restrict__ logits,
                                                              float *__restrict__ low, int T, float eps, int exact_all,
                                                              int32_t *__restrict__ ids, float *__restrict__ weights,
                                                              omni_sort_state st, const char *prefetch, int prefetch_pieces) {
    __shared__ ExactScratch scratch;
    __shared__ int s_flag;
    if (PREFETCH) prefetch_share(prefetch, prefetch_pieces);
    dep_wait();
    dep_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long row = blockIdx.x;
    if (row >= T) return;                                  // blocks that only ask for weights
    const uint4 xq = recheck_x(xn, row, lane, warp);
    float v[4];
    if (warp < 2)
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = logits[row * OMNI_E + lane + 32 * j];
    if (warp == 1) recheck_list(v, eps, lane, scratch);    // beside the selection, in case the row is too close
    if (warp == 0) {
        bool bad = false;
        float max_abs = 0.f;
        uint32_t key[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            bad |= !(fabsf(v[j]) < CUDART_INF_F);
            max_abs = fmaxf(max_abs, fabsf(v[j]));
            key[j] = ranking_key(v[j], lane + 32 * j);
        }
        bool close = false;
        if (__any_sync(FULL, bad)) {
            write_fallback(lane, ids, weights, row, st.status);
        } else {
            max_abs = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(max_abs)));      // not negative: ordered like its bits
            float tv[9];
            int my_id = 0;
#pragma unroll
            for (int r = 0; r < 9; r++) {
                const uint32_t top = __reduce_max_sync(FULL, max(max(key[0], key[1]), max(key[2], key[3])));
                const int id = ranked_expert(top), j = id >> 5;
                tv[r] = __shfl_sync(FULL, j == 0 ? v[0] : j == 1 ? v[1] : j == 2 ? v[2] : v[3], id & 31);
                if (lane == r) my_id = id;
#pragma unroll
                for (int jj = 0; jj < 4; jj++) if (key[jj] == top) key[jj] = 0;
            }
            close = exact_all != 0 || near_tie(tv, eps, max_abs);
            if (!close) {
                float mine = tv[0];
#pragma unroll
                for (int k = 1; k < 8; k++) if (lane == k) mine = tv[k];
                const float p = expf(mine - tv[0]);
                float sum = 0.f;
#pragma unroll
                for (int k = 0; k < 8; k++) sum += __shfl_sync(FULL, p, k);
                const float inv = 1.f / sum;
                if (lane < 8) { ids[row * 8 + lane] = my_id; weights[row * 8 + lane] = p * inv; }
            } else if (lane == 0) {
                atomicAdd(st.n_flag, 1);
            }
        }
        if (lane == 0) s_flag = close;
    }
    __syncthreads();
    if (s_flag)
        recheck_row(xq, w, bias, logits, low, row, ids, weights, nullptr, st.status, scratch, lane, warp, [] { __syncthreads(); });
    __syncthreads();                                       // s_flag has been read by all
    if (T > 1) {                                           // a single block needs no count
        if (warp == 0) {
            __threadfence();                               // this row's ids, in front of the count
            __syncwarp();
            if (lane == 0) s_flag = atomicAdd(st.n_flag + 2, 1) == T - 1;
        }
        __syncthreads();
        if (!s_flag) return;
        __threadfence();
    }

    // ---- the last block: counting sort of all assignments.  A token's experts are distinct, so the tokens of
    // a segment that chose an expert are a mask of 32 bits and a token's rank among them is a count of bits.
    __shared__ unsigned mask[ROUTE_SEGS][OMNI_E];
    __shared__ int base[ROUTE_SEGS][OMNI_E];
    __shared__ ExpertScan scan;
    const int nseg = (T + 31) / 32;
    for (int i = threadIdx.x; i < nseg * OMNI_E; i += EXACT_THREADS) mask[0][i] = 0;
    if (threadIdx.x == 0) st.n_flag[2] = 0;
    constexpr int PER = (ROUTE_SEGS + EXACT_WARPS - 1) / EXACT_WARPS;
    int4 lo[PER], hi[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int t = (warp + i * EXACT_WARPS) * 32 + lane;
        if (t < T) { lo[i] = __ldcg(reinterpret_cast<const int4 *>(ids) + 2 * t); hi[i] = __ldcg(reinterpret_cast<const int4 *>(ids) + 2 * t + 1); }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int s = warp + i * EXACT_WARPS;
        if (s * 32 + lane < T) {
            unsigned *m = mask[s];
            const unsigned bit = 1u << lane;
            atomicOr(m + lo[i].x, bit); atomicOr(m + lo[i].y, bit); atomicOr(m + lo[i].z, bit); atomicOr(m + lo[i].w, bit);
            atomicOr(m + hi[i].x, bit); atomicOr(m + hi[i].y, bit); atomicOr(m + hi[i].z, bit); atomicOr(m + hi[i].w, bit);
        }
    }
    __syncthreads();
    int total = 0;
    const int e128 = threadIdx.x & (OMNI_E - 1);
#pragma unroll 4
    for (int s = 0; s < nseg; s++) {
        if (threadIdx.x < OMNI_E) base[s][e128] = total;
        total += __popc(mask[s][e128]);
    }
    const int off = scan_experts(scan, total, st, true);
    __shared__ int offs[OMNI_E];
    if (threadIdx.x < OMNI_E) offs[threadIdx.x] = off;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int s = warp + i * EXACT_WARPS, t = s * 32 + lane;
        if (t < T) {
            const unsigned lt = (1u << lane) - 1u;
            auto place = [&](int e) {
                const int r = offs[e] + base[s][e] + __popc(mask[s][e] & lt);
                st.rowmap[r] = t;
                return r;
            };
            const int4 a = make_int4(place(lo[i].x), place(lo[i].y), place(lo[i].z), place(lo[i].w));
            const int4 b = make_int4(place(hi[i].x), place(hi[i].y), place(hi[i].z), place(hi[i].w));
            reinterpret_cast<int4 *>(st.slots)[2 * t] = a;
            reinterpret_cast<int4 *>(st.slots)[2 * t + 1] = b;
        }
    }
}

// ------------------------------------------------------------------ start of a pass
// Clears the status word, the flagged-row count that a pass which failed between the router and the sort leaves
// behind and, with expert parallelism, the bucket counters.  One kernel of the chain: as memset nodes these
// cost 3.5 us each, and the kernel behind a memset starts without an overlap.
__global__ void __launch_bounds__(OMNI_EP_BUCKETS) begin_kernel(uint32_t *status, int32_t *n_flag, int32_t *buckets) {
    dep_wait();
    dep_launch();
    if (threadIdx.x == 0) { *status = 0; *n_flag = 0; }
    if (buckets) buckets[threadIdx.x] = 0;
}

// ------------------------------------------------------------------ gather (permute rows)
// xg[row] = xn[rowmap[row]]: 4 KiB per row, one warp per row, 16-byte lanes.
__global__ void __launch_bounds__(256) gather_kernel(const uint4 *__restrict__ xn, const int32_t *__restrict__ rowmap,
                                                     int rows8, uint4 *__restrict__ xg) {
    dep_wait();
    dep_launch();
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * 8;
    for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < rows8; r += warps) {
        const long t = rowmap[r];
        const uint4 *src = xn + t * (OMNI_H / 8);
        uint4 *dst = xg + (long)r * (OMNI_H / 8);
        uint4 v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __ldg(src + lane + 32 * i);
#pragma unroll
        for (int i = 0; i < 8; i++) dst[lane + 32 * i] = v[i];
    }
}

// ------------------------------------------------------------------ RMSNorm in front of the block
// xn[t] = bf16( x[t] * rsqrt(mean(x[t]^2) + eps) * w )  (metal/clef.metal:190-204, `rmsnorm_f32`;
// the product order (x * inv) * w is the reference's).  One block per token, eight elements per
// thread: 8 KiB read, 4 KiB written per row.
__global__ void __launch_bounds__(256) rmsnorm_bf16_kernel(const float4 *__restrict__ x, const float4 *__restrict__ w,
                                                           float eps, uint4 *__restrict__ xn) {
    __shared__ float part[8];
    dep_wait();
    dep_launch();
    const long t = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float4 a = x[t * (OMNI_H / 4) + threadIdx.x * 2], b = x[t * (OMNI_H / 4) + threadIdx.x * 2 + 1];
    const float4 wa = __ldg(w + threadIdx.x * 2), wb = __ldg(w + threadIdx.x * 2 + 1);
    float ss = a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w + b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) ss += __shfl_xor_sync(FULL, ss, s);
    if (lane == 0) part[warp] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) tot += part[i];                 // same order in every thread
    const float inv = 1.0f / sqrtf(tot / (float)OMNI_H + eps);
    const __nv_bfloat162 p0 = __floats2bfloat162_rn(__fmul_rn(__fmul_rn(a.x, inv), wa.x), __fmul_rn(__fmul_rn(a.y, inv), wa.y));
    const __nv_bfloat162 p1 = __floats2bfloat162_rn(__fmul_rn(__fmul_rn(a.z, inv), wa.z), __fmul_rn(__fmul_rn(a.w, inv), wa.w));
    const __nv_bfloat162 p2 = __floats2bfloat162_rn(__fmul_rn(__fmul_rn(b.x, inv), wb.x), __fmul_rn(__fmul_rn(b.y, inv), wb.y));
    const __nv_bfloat162 p3 = __floats2bfloat162_rn(__fmul_rn(__fmul_rn(b.z, inv), wb.z), __fmul_rn(__fmul_rn(b.w, inv), wb.w));
    uint4 o;
    o.x = *reinterpret_cast<const uint32_t *>(&p0); o.y = *reinterpret_cast<const uint32_t *>(&p1);
    o.z = *reinterpret_cast<const uint32_t *>(&p2); o.w = *reinterpret_cast<const uint32_t *>(&p3);
    xn[t * (OMNI_H / 8) + threadIdx.x] = o;
}

// ------------------------------------------------------------------ combine
constexpr int DISCARD_MIN = 448, DISCARD_MAX = 2560;     // tokens
// x[t] += sum over the token's experts in ascending expert id of w * d[slot]
// (clef.metal:2504-2521: fixed order, separate multiply and add, residual added once).
// HBM bound: 32 KiB of d and 16 KiB of x per token.  DISCARD: d is dead once it has been read, and what of it is still in L2 then
// need not go to memory (up to 32 KiB per token that compete with the weights of the next pass).  The line, in tokens for the 126 MB of L2 of the one
// device this is built for: up to 448 tokens it gains nothing and costs nothing, above 2560 (84 MB) part of d has left L2 before it is read, and
// discarding such lines costs.  us per block, without and with, each alone under its own clock, on two GPUs: 400 tokens 213.0 -> 212.8, 448 208.3 -> 208.1,
// 511 218.6 -> 217.4 and 211.5 -> 210.0, 1030 237.0 -> 234.7 and 228.6 -> 223.9, 1536 258.6 -> 253.6 and 246.7 -> 242.0, 2048 280.5 -> 276.7 and
// 266.5 -> 261.7, 2500 301.2 -> 299.1, 2560 286.8 -> 283.9; beyond: 3000 327.7 -> 328.6, 4096 between 1.1 % faster and 0.8 % slower, 16384 2 % slower.
template <bool DISCARD>
__global__ void __launch_bounds__(256) combine_kernel(const uint4 *__restrict__ d, const int32_t *__restrict__ ids,
                                                      const float *__restrict__ weights,
                                                      const int32_t *__restrict__ slots, float *__restrict__ x) {
    dep_wait();
    dep_launch();
    const long t = blockIdx.x;
    // the residual does not depend on the routing: its loads travel with the routing's
    float4 *xp = reinterpret_cast<float4 *>(x + t * OMNI_H) + threadIdx.x * 2;
    float4 a = xp[0], b = xp[1];
    int id[8], sl[8]; float w[8];
    {
        const int4 i0 = __ldg(reinterpret_cast<const int4 *>(ids + t * 8)), i1 = __ldg(reinterpret_cast<const int4 *>(ids + t * 8) + 1);
        const int4 s0 = __ldg(reinterpret_cast<const int4 *>(slots + t * 8)), s1 = __ldg(reinterpret_cast<const int4 *>(slots + t * 8) + 1);
        const float4 w0 = __ldg(reinterpret_cast<const float4 *>(weights + t * 8)), w1 = __ldg(reinterpret_cast<const float4 *>(weights + t * 8) + 1);
        id[0] = i0.x; id[1] = i0.y; id[2] = i0.z; id[3] = i0.w; id[4] = i1.x; id[5] = i1.y; id[6] = i1.z; id[7] = i1.w;
        sl[0] = s0.x; sl[1] = s0.y; sl[2] = s0.z; sl[3] = s0.w; sl[4] = s1.x; sl[5] = s1.y; sl[6] = s1.z; sl[7] = s1.w;
        w[0] = w0.x; w[1] = w0.y; w[2] = w0.z; w[3] = w0.w; w[4] = w1.x; w[5] = w1.y; w[6] = w1.z; w[7] = w1.w;
    }
    // stable insertion sort by expert id (ids of one token are distinct on a valid route)
#pragma unroll
    for (int i = 1; i < 8; i++) {
#pragma unroll
        for (int j = i; j > 0; j--) {
            if (id[j - 1] > id[j]) {
                int ti = id[j]; id[j] = id[j - 1]; id[j - 1] = ti;
                int ts = sl[j]; sl[j] = sl[j - 1]; sl[j - 1] = ts;
                float tw = w[j]; w[j] = w[j - 1]; w[j - 1] = tw;
            }
        }
    }
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; j++) acc[j] = 0.f;
    uint4 q8[8];
#pragma unroll
    for (int k = 0; k < 8; k++) q8[k] = __ldcs(d + (long)sl[k] * (OMNI_H / 8) + threadIdx.x);   // each row is read once
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const uint4 q = q8[k];
        const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            acc[2 * j] = __fadd_rn(acc[2 * j], __fmul_rn(bf16_bits_to_float(u[j] & 0xffffu), w[k]));
            acc[2 * j + 1] = __fadd_rn(acc[2 * j + 1], __fmul_rn(bf16_bits_to_float(u[j] >> 16), w[k]));
        }
    }
    a.x += acc[0]; a.y += acc[1]; a.z += acc[2]; a.w += acc[3];
    b.x += acc[4]; b.y += acc[5]; b.z += acc[6]; b.w += acc[7];
    xp[0] = a; xp[1] = b;
    if (DISCARD) {
        // the warp has read its 512 bytes of the eight rows: four lines each, a lane per line
        __syncwarp();
        const int lane = threadIdx.x & 31;
        int row = sl[0];
#pragma unroll
        for (int k = 1; k < 8; k++) if (lane >> 2 == k) row = sl[k];
        asm volatile("discard.global.L2 [%0], 128;" ::"l"(d + (long)row * (OMNI_H / 8) + (threadIdx.x & ~31) + (lane & 3) * 8) : "memory");
    }
}

// ------------------------------------------------------------------ CUDA-core check kernels for the expert products
__device__ __forceinline__ int expert_of_row(const int32_t *offsets, int row) {
    int lo = 0, hi = OMNI_E;            // largest e with offsets[e] <= row (upper bound, clef.metal:2466-2471)
    while (lo + 1 < hi) { const int mid = (lo + hi) >> 1; if (offsets[mid] <= row) lo = mid; else hi = mid; }
    return lo;
}

// block = one permuted row x 128 of the 768 intermediate columns
__global__ void __launch_bounds__(128) gateup_simple_kernel(const __nv_bfloat16 *__restrict__ xg,
                                                            const __nv_bfloat16 *__restrict__ gate_up,
                                                            const int32_t *__restrict__ offsets,
                                                            __nv_bfloat16 *__restrict__ h) {
    __shared__ float xs[OMNI_H];
    const long row = blockIdx.x;
    if (row >= offsets[OMNI_E]) return;
    const int e = expert_of_row(offsets, (int)row);
    for (int k = threadIdx.x; k < OMNI_H; k += 128) xs[k] = __bfloat162float(xg[row * OMNI_H + k]);
    __syncthreads();
    const int f = blockIdx.y * 128 + threadIdx.x;
    const uint4 *gr = reinterpret_cast<const uint4 *>(gate_up + ((long)e * 2 * OMNI_F + f) * OMNI_H);
    const uint4 *ur = reinterpret_cast<const uint4 *>(gate_up + ((long)e * 2 * OMNI_F + OMNI_F + f) * OMNI_H);
    float g = 0.f, u = 0.f;
    for (int k8 = 0; k8 < OMNI_H / 8; k8++) {
        const uint4 a = __ldg(gr + k8), b = __ldg(ur + k8);
        const uint32_t au[4] = {a.x, a.y, a.z, a.w}, bu[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            g = fmaf(xs[k8 * 8 + 2 * j], bf16_bits_to_float(au[j] & 0xffffu), g);
            g = fmaf(xs[k8 * 8 + 2 * j + 1], bf16_bits_to_float(au[j] >> 16), g);
            u = fmaf(xs[k8 * 8 + 2 * j], bf16_bits_to_float(bu[j] & 0xffffu), u);
            u = fmaf(xs[k8 * 8 + 2 * j + 1], bf16_bits_to_float(bu[j] >> 16), u);
        }
    }
    h[row * OMNI_F + f] = __float2bfloat16(g / (1.f + expf(-g)) * u);
}

// block = one permuted row x 128 of the 2048 output columns
__global__ void __launch_bounds__(128) down_simple_kernel(const __nv_bfloat16 *__restrict__ h,
                                                          const __nv_bfloat16 *__restrict__ down,
                                                          const int32_t *__restrict__ offsets,
                                                          __nv_bfloat16 *__restrict__ d) {
    __shared__ float hs[OMNI_F];
    const long row = blockIdx.x;
    if (row >= offsets[OMNI_E]) return;
    const int e = expert_of_row(offsets, (int)row);
    for (int k = threadIdx.x; k < OMNI_F; k += 128) hs[k] = __bfloat162float(h[row * OMNI_F + k]);
    __syncthreads();
    const int c = blockIdx.y * 128 + threadIdx.x;
    const uint4 *wr = reinterpret_cast<const uint4 *>(down + ((long)e * OMNI_H + c) * OMNI_F);
    float acc = 0.f;
    for (int k8 = 0; k8 < OMNI_F / 8; k8++) {
        const uint4 a = __ldg(wr + k8);
        const uint32_t au[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            acc = fmaf(hs[k8 * 8 + 2 * j], bf16_bits_to_float(au[j] & 0xffffu), acc);
            acc = fmaf(hs[k8 * 8 + 2 * j + 1], bf16_bits_to_float(au[j] >> 16), acc);
        }
    }
    d[row * OMNI_H + c] = __float2bfloat16(acc);
}

// ------------------------------------------------------------------ small utilities
__global__ void fill_u32_kernel(uint32_t *p, uint32_t v, size_t words) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}

__global__ void touch_kernel(const uint32_t *p, uint32_t *sink) {
    if (p[0] == 0x7fc00001u && sink) *sink = 1;    // read-only touch (clef_metal_omni.m:138-147)
}

// Layer-major capture rows: logits[128], low[128], ids[8], weights[8] = 1088 bytes.  `low` is the
// remainder of the logits the exact pass evaluated and zero for the others.
struct TraceRow { float logits[OMNI_E], low[OMNI_E]; int32_t ids[OMNI_TOP]; float weights[OMNI_TOP]; };

__global__ void trace_kernel(const float *__restrict__ logits, const float *__restrict__ low, const int32_t *__restrict__ ids,
                             const float *__restrict__ weights, int rows, int start, int first, int captured, int layer,
                             TraceRow *__restrict__ out) {
    const int p = blockIdx.x;                 // chunk-local row
    const int row = start + p - first;
    if (p >= rows || row < 0 || row >= captured) return;
    TraceRow &r = out[(long)layer * captured + row];
    const int e = threadIdx.x;
    r.logits[e] = logits[(long)p * OMNI_E + e];
    r.low[e] = low[(long)p * OMNI_E + e];
    if (e < 8) { r.ids[e] = ids[(long)p * 8 + e]; r.weights[e] = weights[(long)p * 8 + e]; }
}

}  // namespace

// ====================================================================== launchers
extern "C" {

// Process-wide switch for programmatic dependent launch of the pass's kernel chain.
static int g_dependent_launch = 1;
int omni_dependent_launch_enabled(void) { return g_dependent_launch; }
void omni_set_dependent_launch(int on) { g_dependent_launch = on != 0; }

cudaError_t omni_launch_router_simple(const void *xn, const void *router, const float *bias, int T, float *logits,
                                      cudaStream_t s) {
    router_simple_kernel<<<T, 128, 0, s>>>((const __nv_bfloat16 *)xn, (const __nv_bfloat16 *)router, bias, logits);
    return cudaGetLastError();
}

cudaError_t omni_launch_select(const float *logits, int T, float eps, int exact_all, int32_t *ids, float *weights,
                               int32_t *flag_rows, int32_t *n_flag, uint32_t *status, cudaStream_t s) {
    select_kernel<<<(T + 7) / 8, 256, 0, s>>>(logits, T, eps, exact_all, ids, weights, flag_rows, n_flag, status);
    return cudaGetLastError();
}

cudaError_t omni_launch_recheck(int32_t *segcount, const void *xn, const void *router, const float *bias, float *logits,
                                float *low, const int32_t *flag_rows, const int32_t *n_flag, int T, float eps, int32_t *ids,
                                float *weights, uint32_t *status, const void *prefetch, size_t prefetch_bytes, int n_sm, cudaStream_t s) {
    int blocks = T < n_sm * 8 ? T : n_sm * 8;
    const int pieces = (int)(prefetch_bytes / OMNI_PREFETCH_PIECE);
    if (pieces && blocks < n_sm) blocks = n_sm;
    return omni_launch_chain(pieces ? recheck_kernel<true> : recheck_kernel<false>, dim3(blocks), dim3(EXACT_THREADS), 0, s, (const __nv_bfloat16 *)xn,
                             (const __nv_bfloat16 *)router, bias, logits, low, flag_rows, n_flag, T, eps, ids, weights, segcount, status,
                             (const char *)prefetch, pieces);
}

// sort state: n_flag[0] counts the flagged rows, n_flag[2] the blocks that are done
cudaError_t omni_launch_route(const void *xn, const void *router, const float *bias, float *logits, float *low, int T, float eps,
                              int exact_all, int32_t *ids, float *weights, omni_sort_state st, const void *prefetch,
                              size_t prefetch_bytes, int n_sm, cudaStream_t s) {
    if (T > OMNI_ROUTE_MAX_ROWS) return cudaErrorInvalidValue;
    const int pieces = (int)(prefetch_bytes / OMNI_PREFETCH_PIECE);
    return omni_launch_chain(pieces ? route_kernel<true> : route_kernel<false>, dim3(pieces && T < n_sm ? n_sm : T), dim3(EXACT_THREADS), 0, s,
                             (const __nv_bfloat16 *)xn, (const __nv_bfloat16 *)router, bias, logits, low, T, eps, exact_all, ids, weights, st,
                             (const char *)prefetch, pieces);
}

cudaError_t omni_launch_begin(uint32_t *status, int32_t *n_flag, int32_t *buckets, cudaStream_t s) {
    return omni_launch_chain(begin_kernel, dim3(1), dim3(OMNI_EP_BUCKETS), 0, s, status, n_flag, buckets);
}

cudaError_t omni_launch_router_exact(const void *xn, const void *router, const float *bias, int T, double *logits,
                                     cudaStream_t s) {
    router_exact_kernel<<<T, 128, 0, s>>>((const __nv_bfloat16 *)xn, (const __nv_bfloat16 *)router, bias, logits);
    return cudaGetLastError();
}

cudaError_t omni_launch_route_pairs(const float *hi, const float *lo, int rows, int32_t *ids, float *weights,
                                    uint32_t *status, cudaStream_t s) {
    route_pairs_kernel<<<(rows + 7) / 8, 256, 0, s>>>(hi, lo, rows, ids, weights, status);
    return cudaGetLastError();
}

cudaError_t omni_launch_assign(const int32_t *ids, int rows, omni_sort_state st, int have_counts, cudaStream_t s) {
    const int A = rows * OMNI_TOP;
    const int nseg = (A + OMNI_SEG - 1) / OMNI_SEG;
    const int blocks = (nseg + 7) / 8;
    cudaError_t e = cudaSuccess;
    if (!have_counts) e = omni_launch_chain(assign_hist_kernel, dim3(blocks), dim3(256), 0, s, ids, A, nseg, st.segcount, st.status);
    if (e == cudaSuccess)
        e = omni_launch_chain(assign_kernel, dim3((nseg + ASSIGN_SEGS - 1) / ASSIGN_SEGS), dim3(ASSIGN_THREADS), 0, s, ids, A, nseg, st);
    return e;
}

cudaError_t omni_launch_gather(const void *xn, const int32_t *rowmap, int rows8, void *xg, cudaStream_t s) {
    int blocks = (rows8 + 7) / 8;
    if (blocks > 148 * 16) blocks = 148 * 16;
    return omni_launch_chain(gather_kernel, dim3(blocks), dim3(256), 0, s, (const uint4 *)xn, rowmap, rows8, (uint4 *)xg);
}

cudaError_t omni_launch_rmsnorm(const float *x, const float *w, float eps, int rows, void *xn, cudaStream_t s) {
    return omni_launch_chain(rmsnorm_bf16_kernel, dim3(rows), dim3(256), 0, s, (const float4 *)x, (const float4 *)w, eps, (uint4 *)xn);
}

cudaError_t omni_launch_combine(const void *d, const int32_t *ids, const float *weights, const int32_t *slots,
                                float *x, int T, int dead, cudaStream_t s) {
    return omni_launch_chain(dead && T >= DISCARD_MIN && T <= DISCARD_MAX ? combine_kernel<true> : combine_kernel<false>, dim3(T), dim3(256), 0, s, (const uint4 *)d, ids, weights, slots, x);
}

cudaError_t omni_launch_gateup_simple(const void *xg, const void *gate_up, const int32_t *offsets, int rows8, void *h,
                                      cudaStream_t s) {
    gateup_simple_kernel<<<dim3(rows8, OMNI_F / 128), 128, 0, s>>>((const __nv_bfloat16 *)xg,
                                                                   (const __nv_bfloat16 *)gate_up, offsets,
                                                                   (__nv_bfloat16 *)h);
    return cudaGetLastError();
}

cudaError_t omni_launch_down_simple(const void *h, const void *down, const int32_t *offsets, int rows8, void *d,
                                    cudaStream_t s) {
    down_simple_kernel<<<dim3(rows8, OMNI_H / 128), 128, 0, s>>>((const __nv_bfloat16 *)h, (const __nv_bfloat16 *)down,
                                                                 offsets, (__nv_bfloat16 *)d);
    return cudaGetLastError();
}

cudaError_t omni_launch_fill_u32(void *p, uint32_t v, size_t words, cudaStream_t s) {
    if (!words) return cudaSuccess;
    size_t blocks = (words + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    fill_u32_kernel<<<(unsigned)blocks, 256, 0, s>>>((uint32_t *)p, v, words);
    return cudaGetLastError();
}

cudaError_t omni_launch_touch(const void *p, uint32_t *sink, cudaStream_t s) {
    touch_kernel<<<1, 1, 0, s>>>((const uint32_t *)p, sink);
    return cudaGetLastError();
}

cudaError_t omni_launch_trace(const float *logits, const float *low, const int32_t *ids, const float *weights, int rows, int start,
                              int first, int captured, int layer, void *trace, cudaStream_t s) {
    trace_kernel<<<rows, OMNI_E, 0, s>>>(logits, low, ids, weights, rows, start, first, captured, layer, (TraceRow *)trace);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- assignment without allocation
// Scratch of the sort (segment histograms, tile list, counters) for at most
// CLEF_OMNI_NOALLOC_MAX_ROWS tokens, reserved in the module image: about 72 KB on every GPU
// that loads the library, for the life of the process.
namespace {
constexpr int NOALLOC_MAX_ROWS = 4096;
constexpr int NOALLOC_MAX_SEGS = NOALLOC_MAX_ROWS * OMNI_TOP / OMNI_SEG;
struct NoAllocScratch {
    int32_t segcount[NOALLOC_MAX_SEGS * OMNI_E];
    omni_ttile ttiles[NOALLOC_MAX_ROWS * OMNI_TOP / OMNI_TILE_N + OMNI_E];
    int32_t n_ttiles, sched[8];
    uint32_t status;
    int32_t n_flag[2];
};
static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoAllocScratch)];
// Device address of the array above, per device.  In host code the symbol's name is only a
// stand-in; the usable address comes from cudaGetSymbolAddress with that device current.
static NoAllocScratch *g_noalloc_ptr[64];
}  // namespace

cudaError_t omni_noalloc_assign(const int32_t *ids, int rows, int32_t *counts, int32_t *offsets, int32_t *rowmap,
                                int32_t *slots, uint32_t *status, cudaStream_t s, int *max_rows) {
    if (max_rows) *max_rows = NOALLOC_MAX_ROWS;
    if (rows <= 0 || rows > NOALLOC_MAX_ROWS) return cudaErrorInvalidValue;
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_ptr[dev] = static_cast<NoAllocScratch *>(p);
    }
    NoAllocScratch *sc = g_noalloc_ptr[dev];
    if (!status) {
        // No word of the caller's to report into: the bad-id bit then lands in the shared scratch
        // word, which no entry point reads back, and the id is sorted as id & 127 (documented in
        // the header).  The word keeps whatever the previous call left: start it at zero.
        e = cudaMemsetAsync(&sc->status, 0, sizeof(uint32_t), s);
        if (e != cudaSuccess) return e;
        status = &sc->status;
    }
    omni_sort_state st;
    st.counts = counts; st.offsets = offsets; st.rowmap = rowmap; st.slots = slots;
    st.segcount = sc->segcount; st.ttiles = sc->ttiles; st.n_ttiles = &sc->n_ttiles; st.sched = sc->sched;
    st.status = status;
    st.n_flag = sc->n_flag;
    st.longest_first = 0; st.tile_n = OMNI_TILE_N;
    return omni_launch_assign(ids, rows, st, 0, s);
}

}  // extern "C"
