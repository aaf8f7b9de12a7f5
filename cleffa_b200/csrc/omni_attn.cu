// Attention half of a Clef-Omni decoder layer on sm_100a: the step in front of the MoE block.
//   attn_prep_kernel    per-head RMS norm of q and k, interleaved three-axis rotary, values transposed, q/k/v
//                       laid out per head (reference: metal/clef.metal:2073-2130, omni_attn_prep)
//   attention_kernel    causal grouped-query attention inside each record of the packed batch,
//                       online softmax (reference: metal/clef.metal:2174-2319, omni_attention)
//
// Both products of the attention run on tcgen05 with operands in 128-byte-swizzled shared memory and
// accumulators in tensor memory.  Key blocks start at the record's first token, so a token sees the same blocks whether
// its record is packed with others or runs alone.  V is kept transposed ([d][token]) so that both
// products read K-major operands; each record's columns start at a multiple of 64 tokens
// (`vcol`), which keeps every TMA box 16-byte aligned.  Every wait is bounded.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "omni_internal.h"
#include "omni_land.cuh"
#include "omni_pair.cuh"
#include "omni_pdl.cuh"
#include "omni_ptx.cuh"

namespace {

constexpr int HD = OMNI_HD, NH = OMNI_NH, NKV = OMNI_NKV;

// ------------------------------------------------------------------ q/k norm + rotary + layout
// Two jobs of one launch that read different columns of the projections: blocks below `prep_blocks` norm and
// rotate q and k, the others transpose v.  As two launches the second waited for the first (3 us at 37
// tokens, 12 at 16384).
//
// Norm and rotary: four warps per token, nine heads each (32 query heads, then the 4 key heads, dealt in turn).  A lane
// holds four consecutive elements of the 128 of a head (one 8-byte load and store); pair p of a
// head is (element p, element p + 64), so a lane's partners sit in lane ^ 16.  The pair's angle is
// position[axis] * theta^(-p/64) with axis = p % 3 for p < 60 and the temporal axis above (sections
// 24/20/20 interleaved; clef.metal:2051-2053).  The angle is formed and reduced modulo 2 pi in
// FP64 -- FP32 loses ~pos * 6e-8 rad (clef.metal:2055-2060) -- from frequencies that binding the layer left in
// `freq` (rope_freq_kernel) instead of an exp2 and a log2 per token and pair.  Cosine and sine are the same for every
// head of the token and computed once per warp (one warp for all heads of a token, which forms them once, was 8 % slower for the
// attention half of 2048 tokens and no faster at 16384: fewer loads in flight).
constexpr int PREP_THREADS = 256, PREP_WARPS = 4, PREP_HEADS = (NH + NKV) / PREP_WARPS;
static_assert((NH + NKV) % PREP_WARPS == 0, "heads are dealt to the warps of a token");

__global__ void __launch_bounds__(PREP_THREADS) attn_prep_kernel(const __nv_bfloat16 *__restrict__ qkv, const float *__restrict__ qw,
                                                                 const float *__restrict__ kw, const int32_t *__restrict__ pos,
                                                                 const double *__restrict__ freq, const int32_t *__restrict__ vcol, int T,
                                                                 int prep_blocks, int head_stride, int vpitch, float eps,
                                                                 __nv_bfloat16 *__restrict__ Q, __nv_bfloat16 *__restrict__ K,
                                                                 __nv_bfloat16 *__restrict__ Vt, uint32_t *__restrict__ status) {
    __shared__ unsigned short tile[64][HD + 2];
    __shared__ int col[64];
    dep_wait();
    dep_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool bad = false;
    if ((int)blockIdx.x >= prep_blocks) {
        // Values, transposed: Vt[kh][d][column of the token].  One block per (64 tokens, key/value head):
        // rows read whole (256 bytes per token), written as 64-token runs per head dimension.
        const int vb = blockIdx.x - prep_blocks, t0 = vb / NKV * 64, kh = vb % NKV;
        if (threadIdx.x < 64) col[threadIdx.x] = t0 + threadIdx.x < T ? __ldg(vcol + t0 + threadIdx.x) : -1;
#pragma unroll
        for (int i = warp; i < 64; i += PREP_THREADS / 32) {
            const long t = t0 + i;
            if (t < T) {
                const uint2 v = *reinterpret_cast<const uint2 *>(qkv + t * OMNI_QKV + (long)(NH + NKV + kh) * HD + lane * 4);
                const unsigned short e[4] = {(unsigned short)(v.x & 0xffff), (unsigned short)(v.x >> 16), (unsigned short)(v.y & 0xffff), (unsigned short)(v.y >> 16)};
#pragma unroll
                for (int k = 0; k < 4; k++) { bad |= (e[k] & 0x7f80) == 0x7f80; tile[i][lane * 4 + k] = e[k]; }
            }
        }
        // A nonfinite value fails the pass and is written as zero: a record's last key block of 128 reaches past its own columns,
        // where whatever an earlier batch has left is multiplied by probabilities of zero.  (Attention half of 4096 tokens: this way
        // as before, 1.2 % slower with a choice per element above, 2.4 % with zeros written behind every record.)
        if (__syncthreads_or(bad)) {
            for (int i = warp; i < 64; i += PREP_THREADS / 32)
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if ((tile[i][lane + 32 * k] & 0x7f80) == 0x7f80) tile[i][lane + 32 * k] = 0;
            __syncthreads();
        }
        unsigned short *out = reinterpret_cast<unsigned short *>(Vt) + (long)kh * HD * vpitch;
        for (int d = warp; d < HD; d += PREP_THREADS / 32)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int i = lane + 32 * k;
                if (col[i] >= 0) out[(long)d * vpitch + col[i]] = tile[i][d];
            }
        if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(status, OMNI_ST_ATTN_NONFINITE);
        return;
    }
    const long t = (long)blockIdx.x * (PREP_THREADS / 32 / PREP_WARPS) + warp / PREP_WARPS;
    if (t >= T) return;
    const int sub = warp % PREP_WARPS;
    const bool upper = lane >= 16;                                               // elements 64..127: the second of each pair
    const __nv_bfloat16 *row = qkv + t * OMNI_QKV + 4 * lane;
    uint2 raw[PREP_HEADS];                                // the loads of all nine heads are in flight together
#pragma unroll
    for (int i = 0; i < PREP_HEADS; i++) raw[i] = *reinterpret_cast<const uint2 *>(row + (long)(sub + PREP_WARPS * i) * HD);
    // the four pairs of a lane are those of lane ^ 16 too: each computes two and they swap
    float cs[4], sn[4];
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const int own = (upper ? 2 : 0) + j, pair = 4 * (lane & 15) + own, axis = pair < 60 ? pair % 3 : 0;
        const double angle = (double)__ldg(pos + 3 * t + axis) * __ldg(freq + pair);
        const double turns = rint(angle * 0.15915494309189535);
        const float r = (float)fma(-turns, 6.283185307179586, angle);           // |r| <= pi, accurate to FP32 rounding
        float sj, cj;
        sincosf(r, &sj, &cj);
        const float so = __shfl_xor_sync(0xffffffffu, sj, 16), co = __shfl_xor_sync(0xffffffffu, cj, 16);
        cs[j] = upper ? co : cj; cs[j + 2] = upper ? cj : co;
        sn[j] = upper ? so : sj; sn[j + 2] = upper ? sj : so;
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (!upper) sn[j] = -sn[j];                                              // lo' = lo cos - hi sin, hi' = hi cos + lo sin
    const float4 wq = __ldg(reinterpret_cast<const float4 *>(qw) + lane), wk = __ldg(reinterpret_cast<const float4 *>(kw) + lane);
#pragma unroll
    for (int i = 0; i < PREP_HEADS; i++) {
        const int h = sub + PREP_WARPS * i;
        const bool query = h < NH;
        float x[4] = {__uint_as_float(raw[i].x << 16), __uint_as_float(raw[i].x & 0xffff0000u), __uint_as_float(raw[i].y << 16),
                      __uint_as_float(raw[i].y & 0xffff0000u)};
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 4; j++) { bad |= !(fabsf(x[j]) < CUDART_INF_F); sum += x[j] * x[j]; }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
        const float inv = rsqrtf(sum / (float)HD + eps);
        const float4 w = query ? wq : wk;
        x[0] = x[0] * inv * w.x; x[1] = x[1] * inv * w.y; x[2] = x[2] * inv * w.z; x[3] = x[3] * inv * w.w;
        uint32_t o[2];
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            const float p0 = __shfl_xor_sync(0xffffffffu, x[j], 16), p1 = __shfl_xor_sync(0xffffffffu, x[j + 1], 16);
            const float y0 = x[j] * cs[j] + p0 * sn[j], y1 = x[j + 1] * cs[j + 1] + p1 * sn[j + 1];
            bad |= !(fabsf(y0) < CUDART_INF_F) || !(fabsf(y1) < CUDART_INF_F);
            const __nv_bfloat162 bb = __floats2bfloat162_rn(y0, y1);
            o[j >> 1] = *reinterpret_cast<const uint32_t *>(&bb);
        }
        __nv_bfloat16 *dst = query ? Q + ((long)h * head_stride + t) * HD : K + ((long)(h - NH) * head_stride + t) * HD;
        *reinterpret_cast<uint2 *>(dst + 4 * lane) = make_uint2(o[0], o[1]);
    }
    // reported at completion like the reference's status bit 2 (clef.metal:2120)
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(status, OMNI_ST_ATTN_NONFINITE);
}

// theta^(-p/64) of the 64 rotary pairs, once per bound layer
__global__ void rope_freq_kernel(double theta, double *freq) { freq[threadIdx.x] = exp2(-(double)threadIdx.x * (1.0 / 64.0) * log2(theta)); }

// ------------------------------------------------------------------ attention
// Pairs of CTAs that stay resident (clusters of two SMs, tcgen05 cta_group::2) take work items in turn: a pair of
// query heads that share a key/value head and a tile of <= 128 query rows of one record.  Each CTA
// has one of the two heads; a key block of 128 is loaded once for both, half of it into each CTA.
// Key blocks run from the record's start to the tile's diagonal.  For block g of a CTA's sequence:
//   S(g) = Q K^T             tcgen05, FP32, into score buffer g mod 3 of tensor memory
//   P(g) = exp2(c S - m)     by warps of group g mod 3, a thread per query row; BF16, two keys per column,
//                            written over the upper half of the score buffer, which is in registers by then
//   O   += P(g) V            tcgen05 with the A operand read from tensor memory, accumulated over the item's blocks
// With three score buffers the scores of the next two blocks are complete before their softmax begins and
// the value product of a block runs behind the softmax of the next: neither is part of a
// chain from one block to the next.  All that passes from block to block is the row's reference maximum
// m, handed from a group's warp to the next group's warp of the same 32 rows as soon as the block's own
// maximum is known.  (With two heads per CTA and one score buffer each, the chain scores -> softmax -> value
// product -> scores held a block of a head for 1870 cycles, tensor cores and special-function units 55 % busy.)
// m follows the running maximum lazily: only when a block's maximum exceeds it by more than 2^8 is O
// rescaled (in tensor memory, once the previous value product is done); otherwise P simply holds values up to
// 256.  Each group sums its own blocks' probabilities against the m it last saw; the group of the item's
// last block collects the sums, reads O and writes the rows while the others are in the next item.
// The order of every sum goes by the block's place in its own item, so a row's bits do not depend on what the pair
// did before.
struct AttnTile { int32_t rec_start, q0, q_len, vcol0; };          // vcol0: Vt column of the record's first token

constexpr int AT_THREADS = 512;                                    // warp 0 loads, 1 MMA, 2 TMEM, 3 spare, 4..7, 8..11, 12..15 softmax groups 0, 1, 2
constexpr int AT_PAIRS_PER_TILE = NH / 2;                          // work items of a query tile
constexpr int AT_Q_BYTES = 128 * 128 * 2;                          // 32 KiB: 128 rows x 128 BF16 as two 64-column halves
constexpr int AT_KV_BYTES = 64 * 128 * 2;                          // 16 KiB: a CTA's half of a key or value block, as two 64-column halves
constexpr int AT_KV_STAGES = 4, AT_BUFS = 3;
constexpr int AT_TMEM_O = 0, AT_TMEM_S = 128, AT_P_COL = 64;       // O, then three score buffers of 128 columns; P in columns 64..127 of a buffer
constexpr int AT_DATA_BYTES = 2 * AT_Q_BYTES + 2 * AT_KV_STAGES * AT_KV_BYTES;
constexpr int AT_N_BARS = 4 + 4 * AT_KV_STAGES + 3 * AT_BUFS + 1 + 16 + 1;
constexpr int AT_MISC_OFF = AT_DATA_BYTES + AT_N_BARS * 8, AT_XCH_OFF = (AT_MISC_OFF + 64 + 15) & ~15;
constexpr int AT_SMEM_BYTES = AT_XCH_OFF + AT_BUFS * 128 * 4 + 2 * AT_BUFS * 128 * 8 + 1024;
static_assert(AT_SMEM_BYTES <= 232448, "shared memory budget");
constexpr float AT_LAZY = 8.f;                                     // log2 of how far a block may exceed the reference maximum
// 128 registers per thread at launch: 80 do for the first four warps, the softmax threads take 144
constexpr int AT_REGS_FEW = 80, AT_REGS_MANY = 144;
static_assert(128 * AT_REGS_FEW + (AT_THREADS - 128) * AT_REGS_MANY <= AT_THREADS * 128, "registers of the block");

__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D[tmem] (+)= A[tmem] . B[smem]^T over both SMs: A's rows are the TMEM lanes of either CTA, two BF16 of the K extent
// per column.
__device__ __forceinline__ void umma_bf16_ts2(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ float ex2_approx(float x) {          // 2^x, -inf -> 0; relative error ~2^-22, far below BF16's
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// two FP32 lanes per instruction: (a.x * b.x + c.x, a.y * b.y + c.y) and (a.x + b.x, a.y + b.y)
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(*reinterpret_cast<uint64_t *>(&a)), "l"(*reinterpret_cast<uint64_t *>(&b)),
        "l"(*reinterpret_cast<uint64_t *>(&c)));
    return *reinterpret_cast<float2 *>(&d);
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<uint64_t *>(&a)), "l"(*reinterpret_cast<uint64_t *>(&b)));
    return *reinterpret_cast<float2 *>(&d);
}

// The items of one pair of CTAs: the host lists the tiles with the most key blocks first; rounds over the pairs
// alternate in direction, so that no pair gets the longer item of every round.  The entry of the item after the
// current one is on its way meanwhile.
struct AttnItems {
    const AttnTile *tiles;
    int n_items, round;
    int4 cur, ahead;
    __device__ __forceinline__ int index(int r) const {
        const int pairs = (int)gridDim.x >> 1, p = (int)blockIdx.x >> 1;
        return r * pairs + ((r & 1) ? pairs - 1 - p : p);
    }
    __device__ __forceinline__ AttnItems(const AttnTile *t, int n) : tiles(t), n_items(n), round(-1) { fetch(0); }
    __device__ __forceinline__ void fetch(int r) {
        if (index(r) < n_items) ahead = __ldg(reinterpret_cast<const int4 *>(tiles) + index(r) / AT_PAIRS_PER_TILE);
    }
    __device__ __forceinline__ bool more() const { return index(round + 1) < n_items; }
    __device__ __forceinline__ bool next() {
        const bool any = more();
        round++;
        cur = ahead;
        fetch(round + 1);
        return any;
    }
    __device__ __forceinline__ AttnTile tile() const { return AttnTile{cur.x, cur.y, cur.z, cur.w}; }
    __device__ __forceinline__ int h0() const { return 2 * (index(round) % AT_PAIRS_PER_TILE); }            // first query head of the pair
    __device__ __forceinline__ int n_blocks() const { return (cur.y + cur.z - 1 - cur.x) / 128 + 1; }        // from the record's start to the diagonal
};

__global__ void __launch_bounds__(AT_THREADS, 1)
attention_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_vt, const AttnTile *__restrict__ tiles, int n_items, int T, float scale,
                 __nv_bfloat16 *__restrict__ out, int early_dependents, uint32_t *__restrict__ status) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *const smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    auto q_smem = [&](int b) { return smem_base + AT_Q_BYTES * b; };
    auto k_smem = [&](int s) { return smem_base + 2 * AT_Q_BYTES + AT_KV_BYTES * s; };
    auto v_smem = [&](int s) { return smem_base + 2 * AT_Q_BYTES + AT_KV_BYTES * (AT_KV_STAGES + s); };
    const uint32_t bar_base = smem_base + AT_DATA_BYTES;
    auto bar = [&](int i) { return bar_base + 8u * i; };
    // loads are signalled on the first CTA's barriers; what the MMA thread commits arrives in both CTAs
    auto q_full = [&](int b) { return bar(b); };
    auto q_empty = [&](int b) { return bar(2 + b); };
    auto k_full = [&](int s) { return bar(4 + s); };
    auto k_empty = [&](int s) { return bar(4 + AT_KV_STAGES + s); };
    auto v_full = [&](int s) { return bar(4 + 2 * AT_KV_STAGES + s); };
    auto v_empty = [&](int s) { return bar(4 + 3 * AT_KV_STAGES + s); };
    constexpr int B0 = 4 + 4 * AT_KV_STAGES;
    auto s_full = [&](int b) { return bar(B0 + b); };
    auto p_full = [&](int b) { return bar(B0 + AT_BUFS + b); };               // first CTA's: the four warps of the block's group, in both CTAs
    auto pv_done = [&](int b) { return bar(B0 + 2 * AT_BUFS + b); };
    const uint32_t o_empty = bar(B0 + 3 * AT_BUFS);                           // first CTA's: O of the previous item has been read, in both CTAs
    auto fin_full = [&](int q, int slot) { return bar(B0 + 3 * AT_BUFS + 1 + 2 * q + slot); };
    auto fin_empty = [&](int q, int slot) { return bar(B0 + 3 * AT_BUFS + 9 + 2 * q + slot); };
    const uint32_t drain_bar = bar(B0 + 3 * AT_BUFS + 17);
    uint8_t *misc = smem_gen + AT_MISC_OFF;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(misc);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(misc + 4);
    volatile int *armed = reinterpret_cast<volatile int *>(misc + 16);         // [10]: q buffers, k and v stages (parity of the load in flight, -1 none)
    float *m_sh = reinterpret_cast<float *>(smem_gen + AT_XCH_OFF);            // [group][row] reference maximum after the group's block
    float2 *fin = reinterpret_cast<float2 *>(smem_gen + AT_XCH_OFF + AT_BUFS * 128 * 4);   // [slot][group][row] row sum of a group and the maximum it refers to

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = __shfl_sync(0xffffffffu, cluster_ctarank(), 0);
    const bool leader = rank == 0;
    const Abort ab{abort_flag, mapa_u32(bar_base + AT_N_BARS * 8 + 4, rank ^ 1u), status};
    auto lead = [&](uint32_t b) { return mapa_u32(b, 0); };
    auto give = [] { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AT_REGS_FEW)); };

    if (threadIdx.x == 0) {
        for (int i = 0; i < AT_N_BARS; i++) {
            const bool per_warp = (i >= B0 + AT_BUFS && i < B0 + 2 * AT_BUFS) || i == B0 + 3 * AT_BUFS;             // p_full, o_empty
            const bool collect = i >= B0 + 3 * AT_BUFS + 1 && i < B0 + 3 * AT_BUFS + 9;                             // fin_full
            mbar_init(bar(i), per_warp ? 8 : collect ? AT_BUFS - 1 : 1);
        }
        *abort_flag = 0;
        for (int i = 0; i < 2 + 2 * AT_KV_STAGES; i++) armed[i] = -1;
        fence_mbar_init();
        prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_vt);
    }
    cluster_sync_all();                       // the peer's barriers must exist before anything here can signal them
    if (warp == 2) xtmem_alloc<2>(smem_u32((const void *)tmem_slot), 512);
    dep_wait();
    if (early_dependents) dep_launch();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = (uint32_t)uniform_i32((int)*tmem_slot);

    if (warp == 0) {
        // ---------------------------------------------------------- loads of this CTA: its head's Q tile per item; of every block the
        // key rows (head dimensions of V) that are its half.  Keys run ahead of values, as the MMAs do.
        give();
        PipeState pk, pv;
        AttnItems ki(tiles, n_items), vi(tiles, n_items);
        int kj = 0, vj = 0;
        bool ok = true;
        bool k_left = ki.next(), v_left = vi.next();
        auto load_k = [&] {
            if (kj == 0) {
                const int b = ki.round & 1;
                const uint32_t ph = (uint32_t)(ki.round >> 1) & 1u;
                ok = xwait_warp<false>(q_empty(b), ph ^ 1u, ab);
                if (!ok) return;
                if (elect_one()) {
                    if (leader) { armed[b] = (int)ph; mbar_expect_tx(q_full(b), 2 * AT_Q_BYTES); }
                    const int y = (ki.h0() + (int)rank) * T + ki.tile().q0;
                    xtma_2d<2>(q_smem(b), &tm_q, 0, y, lead(q_full(b)), l2_policy_evict_first());                          // d 0..63
                    xtma_2d<2>(q_smem(b) + AT_Q_BYTES / 2, &tm_q, 64, y, lead(q_full(b)), l2_policy_evict_first());         // d 64..127
                }
            }
            ok = xwait_warp<false>(k_empty(pk.stage), pk.phase ^ 1u, ab);
            if (!ok) return;
            if (elect_one()) {
                if (leader) { armed[2 + pk.stage] = (int)pk.phase; mbar_expect_tx(k_full(pk.stage), 2 * AT_KV_BYTES); }
                const int y = ki.h0() / (NH / NKV) * T + ki.tile().rec_start + kj * 128 + (int)rank * 64;
                xtma_2d<2>(k_smem(pk.stage), &tm_k, 0, y, lead(k_full(pk.stage)), l2_policy_evict_last());
                xtma_2d<2>(k_smem(pk.stage) + AT_KV_BYTES / 2, &tm_k, 64, y, lead(k_full(pk.stage)), l2_policy_evict_last());
            }
            pk.advance(AT_KV_STAGES);
            if (++kj == ki.n_blocks()) { kj = 0; k_left = ki.next(); }
        };
        for (int i = 0; i < AT_BUFS && k_left && ok; i++) load_k();
        while (v_left && ok) {
            ok = xwait_warp<false>(v_empty(pv.stage), pv.phase ^ 1u, ab);
            if (!ok) break;
            if (elect_one()) {
                if (leader) { armed[2 + AT_KV_STAGES + pv.stage] = (int)pv.phase; mbar_expect_tx(v_full(pv.stage), 2 * AT_KV_BYTES); }
                const int x = vi.tile().vcol0 + vj * 128, y = vi.h0() / (NH / NKV) * HD + (int)rank * 64;
                xtma_2d<2>(v_smem(pv.stage), &tm_vt, x, y, lead(v_full(pv.stage)), l2_policy_evict_last());                              // keys 0..63 of the block
                xtma_2d<2>(v_smem(pv.stage) + AT_KV_BYTES / 2, &tm_vt, x + 64, y, lead(v_full(pv.stage)), l2_policy_evict_last());
            }
            pv.advance(AT_KV_STAGES);
            if (++vj == vi.n_blocks()) { vj = 0; v_left = vi.next(); }
            if (k_left) load_k();
        }
    } else if (warp == 1 && leader) {
        // ---------------------------------------------------------- MMA issuer
        // Scores run AT_BUFS blocks ahead of value products; behind the value product of block g come the scores of
        // block g + 3 into the buffer it has read P from (the tensor pipe runs them in the order issued).
        give();
        const uint32_t idesc = idesc_bf16(256, 128);
        PipeState pk, pv, bs, bp;                 // stages of K and V; score buffer of the next scores and of the next value product
        AttnItems si(tiles, n_items), pi(tiles, n_items);
        int sj = 0, pj = 0;
        bool ok = true;
        bool s_left = si.next(), p_left = pi.next();
        auto scores = [&] {
            const int b = si.round & 1;
            if (sj == 0) ok = xwait_warp<false>(q_full(b), (uint32_t)(si.round >> 1) & 1u, ab);
            if (ok) ok = xwait_warp<false>(k_full(pk.stage), pk.phase, ab);
            if (!ok) return;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t d = tmem_base + AT_TMEM_S + bs.stage * 128;
#pragma unroll
                for (int half = 0; half < 2; half++) {          // the 128 head dimensions: two 64-wide halves, four K=16 steps each
                    const uint64_t da = smem_desc_sw128(q_smem(b) + half * (AT_Q_BYTES / 2));
                    const uint64_t db = smem_desc_sw128(k_smem(pk.stage) + half * (AT_KV_BYTES / 2));
#pragma unroll
                    for (int k = 0; k < 4; k++) xmma<2>(d, da + 2u * k, db + 2u * k, idesc, (half | k) ? 1u : 0u);
                }
                xcommit<2>(s_full(bs.stage));
                xcommit<2>(k_empty(pk.stage));
                if (sj == si.n_blocks() - 1) xcommit<2>(q_empty(b));
            }
            __syncwarp();
            pk.advance(AT_KV_STAGES);
            bs.advance(AT_BUFS);
            if (++sj == si.n_blocks()) { sj = 0; s_left = si.next(); }
        };
        for (int i = 0; i < AT_BUFS && s_left && ok; i++) scores();
        while (p_left && ok) {
            ok = xwait_warp<false>(v_full(pv.stage), pv.phase, ab);
            if (ok && pj == 0 && pi.round > 0) ok = xwait_warp<false>(o_empty, (uint32_t)(pi.round - 1) & 1u, ab);
            if (ok) ok = xwait_warp<false>(p_full(bp.stage), bp.phase, ab);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t p = tmem_base + AT_TMEM_S + bp.stage * 128 + AT_P_COL;
#pragma unroll
                for (int k = 0; k < 8; k++) {                   // the 128 keys of the block: eight K=16 steps, 8 columns of P each
                    const uint64_t db = smem_desc_sw128(v_smem(pv.stage) + (k >> 2) * (AT_KV_BYTES / 2));
                    umma_bf16_ts2(tmem_base + AT_TMEM_O, p + 8 * k, db + 2u * (k & 3), idesc, (pj | k) ? 1u : 0u);
                }
                xcommit<2>(v_empty(pv.stage));
                xcommit<2>(pv_done(bp.stage));
            }
            __syncwarp();
            pv.advance(AT_KV_STAGES);
            bp.advance(AT_BUFS);
            if (++pj == pi.n_blocks()) { pj = 0; p_left = pi.next(); }
            if (s_left) scores();
        }
        // whatever happened, wait (bounded) until every MMA issued here has retired before tensor memory is released
        if (elect_one()) {
            xcommit<2>(drain_bar);
            const uint64_t t0 = globaltimer_ns();
            while (!mbar_try_wait(drain_bar, 0) && globaltimer_ns() - t0 < WAIT_LIMIT_NS) {}
        }
        __syncwarp();
    } else if (warp < 4) {
        give();
    } else {
        // ---------------------------------------------------------- softmax: a thread per query row
        // The loop runs to its end whatever happens: a warp whose wait ran out does no more work but still meets the
        // others at the barriers below, so none is left in them.
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(AT_REGS_MANY));
        const int grp = (warp - 4) >> 2, q = warp & 3;
        const int r = q * 32 + lane;                                              // row inside the tile = TMEM lane
        const uint32_t tmem_row = tmem_base + ((uint32_t)(q * 32) << 16);
        const float c = scale * 1.4426950408889634f;                              // scores to log2 units
        // named barriers 1 + 4 * group + quadrant: from that group's warp to the next group's
        const int bar_in = 1 + 4 * ((grp + AT_BUFS - 1) % AT_BUFS) + q, bar_out = 1 + 4 * grp + q;
        const float *m_in = m_sh + (grp + AT_BUFS - 1) % AT_BUFS * 128 + r;
        bool alive = true;
        auto wait = [&](uint32_t b, uint32_t parity) {
            if (alive) alive = xwait_warp<false>(b, parity, ab);
        };
        AttnItems it(tiles, n_items);
        int at = 0;                                                               // block of the sequence that the item starts with, mod 3
        uint32_t phase = 0;                                                       // of this group's score buffer
        bool first_ever = true;
        while (it.next()) {
            const int n_blocks = it.n_blocks();
            const int last = (at + n_blocks - 1) % AT_BUFS;                       // group of the item's last block
            const int slot = it.round & 1;
            const uint32_t slot_phase = (uint32_t)(it.round >> 1) & 1u;
            float m = -1e30f, l = 0.f;                                            // this group's sum and the maximum it refers to
            for (int j = (grp + AT_BUFS - at) % AT_BUFS; j < n_blocks; j += AT_BUFS) {
                const bool diagonal = j == n_blocks - 1;                          // the only block with keys after some of the rows
                const uint32_t s_at = tmem_row + AT_TMEM_S + grp * 128;
                uint32_t ta[32], tb[32];
                float bm = -CUDART_INF_F;
                wait(s_full(grp), phase);
                // two sweeps over the row's 128 scores, the maximum first; the upper 64 stay in registers for the second
                auto mask = [&](uint32_t (&v)[32], int key) {
                    if (diagonal) {
#pragma unroll
                        for (int i = 0; i < 32; i++)
                            if (key + i > r) v[i] = 0xff800000u;
                    }
                };
                auto row_max = [&](const uint32_t (&v)[32]) {
                    float a = max3(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2])), b = __uint_as_float(v[3]);
#pragma unroll
                    for (int i = 4; i < 32; i += 4) {
                        a = max3(a, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
                        b = max3(b, __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
                    }
                    bm = max3(bm, a, b);
                };
                if (alive) {
                    tc_fence_after();
                    tmem_ld32(s_at, ta);
                    tmem_ld32(s_at + 32, tb);
                    tmem_ld_wait();
                    mask(ta, 0);
                    row_max(ta);
                    tmem_ld32(s_at + 64, ta);
                    mask(tb, 32);
                    row_max(tb);
                    tmem_ld32(s_at + 96, tb);
                    tmem_ld_wait();
                    mask(ta, 64);
                    row_max(ta);
                    mask(tb, 96);
                    row_max(tb);
                }
                // key 0 of every block is visible to every row (tiles and blocks are both cut from the
                // record's start in steps of 128), so the block maximum is finite
                bm *= c;
                float m_prev = bm;
                if (at + j > 0 || !first_ever) {
                    asm volatile("bar.sync %0, 64;" ::"r"(bar_in) : "memory");
                    if (j > 0) m_prev = *m_in;
                }
                const float m_new = bm > m_prev + AT_LAZY ? bm : m_prev;
                m_sh[grp * 128 + r] = m_new;
                if (!diagonal || it.more()) asm volatile("bar.arrive %0, 64;" ::"r"(bar_out) : "memory");
                if (m_new != m) { l *= ex2_approx(m - m_new); m = m_new; }
                if (__any_sync(0xffffffffu, m_new != m_prev)) {
                    // O may be scaled once the previous block's value product is done; this block's waits for the P below
                    wait(pv_done((grp + AT_BUFS - 1) % AT_BUFS), grp == 0 ? phase ^ 1u : phase);
                    if (alive) {
                        tc_fence_after();
                        const float corr = ex2_approx(m_prev - m_new);
                        for (int o = 0; o < 8; o++) {
                            uint32_t t16[16];
                            tmem_ld16(tmem_row + AT_TMEM_O + o * 16, t16);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 16; i++) t16[i] = __float_as_uint(__uint_as_float(t16[i]) * corr);
                            tmem_st16(tmem_row + AT_TMEM_O + o * 16, t16);
                        }
                    }
                }
                // P = exp2(c s - m) as BF16 (values up to 2^8 while m lags the running maximum), two keys per column
                if (alive) {
                    float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
                    const float2 c2 = make_float2(c, c), nm2 = make_float2(-m_new, -m_new);
                    auto probs = [&](const uint32_t (&v)[32], int piece) {
                        uint32_t pk[16];
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            const float2 e = ffma2(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), c2, nm2);
                            const float2 pp = make_float2(ex2_approx(e.x), ex2_approx(e.y));
                            acc[i & 1] = fadd2(acc[i & 1], pp);
                            const __nv_bfloat162 bb = __floats2bfloat162_rn(pp.x, pp.y);
                            pk[i] = *reinterpret_cast<const uint32_t *>(&bb);
                        }
                        tmem_st16(s_at + AT_P_COL + piece * 16, pk);
                    };
                    probs(ta, 2);
                    tmem_ld32(s_at, ta);
                    probs(tb, 3);
                    tmem_ld32(s_at + 32, tb);
                    tmem_ld_wait();
                    mask(ta, 0);
                    probs(ta, 0);
                    mask(tb, 32);
                    probs(tb, 1);
                    l += (acc[0].x + acc[1].x) + (acc[0].y + acc[1].y);
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote(lead(p_full(grp)));
                }
                phase ^= 1u;
            }
            first_ever = false;
            if (grp != last) {
                wait(fin_empty(q, slot), slot_phase ^ 1u);
                fin[(slot * AT_BUFS + grp) * 128 + r] = make_float2(l, m);
                __syncwarp();
                if (lane == 0) mbar_arrive(fin_full(q, slot));
            } else {
                wait(fin_full(q, slot), slot_phase);
                const float2 f1 = fin[(slot * AT_BUFS + (grp + 1) % AT_BUFS) * 128 + r], f2 = fin[(slot * AT_BUFS + (grp + 2) % AT_BUFS) * 128 + r];
                __syncwarp();
                if (lane == 0) mbar_arrive(fin_empty(q, slot));
                const float lt = l + f1.x * ex2_approx(f1.y - m) + f2.x * ex2_approx(f2.y - m);
                const float inv = lt > 0.f ? 1.f / lt : 0.f;
                wait(pv_done(grp), phase ^ 1u);                                   // the item's last value product
                if (alive) {
                    tc_fence_after();
                    uint4 *dst = reinterpret_cast<uint4 *>(out + (long)(it.tile().q0 + r) * (NH * HD) + (it.h0() + (int)rank) * HD);
#pragma unroll
                    for (int o = 0; o < 4; o++) {
                        uint32_t t32[32];
                        tmem_ld32(tmem_row + AT_TMEM_O + o * 32, t32);
                        tmem_ld_wait();
                        if (o == 3) {                                             // the next item's value products may start
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_remote(lead(o_empty));
                        }
                        if (r < it.tile().q_len) {
#pragma unroll
                            for (int ch = 0; ch < 4; ch++) {
                                uint32_t w[4];
#pragma unroll
                                for (int i = 0; i < 4; i++) {
                                    const __nv_bfloat162 bb = __floats2bfloat162_rn(__uint_as_float(t32[ch * 8 + 2 * i]) * inv,
                                                                                    __uint_as_float(t32[ch * 8 + 2 * i + 1]) * inv);
                                    w[i] = *reinterpret_cast<const uint32_t *>(&bb);
                                }
                                dst[o * 4 + ch] = make_uint4(w[0], w[1], w[2], w[3]);
                            }
                        }
                    }
                }
            }
            at = (at + n_blocks) % AT_BUFS;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0) {
        // a wait ran out; the first CTA knows what both announced
        copies_land(armed, 2 + 2 * AT_KV_STAGES, [&](int i, int parity) {
            const uint32_t b = i < 2 ? q_full(i) : i < 2 + AT_KV_STAGES ? k_full(i - 2) : v_full(i - 2 - AT_KV_STAGES);
            return mbar_try_wait(b, (uint32_t)parity) != 0;
        }, globaltimer_ns, LAND_LIMIT_NS, LAND_SETTLE_NS);
    }
    // neither CTA may leave while the other's MMAs can still read its shared memory
    cluster_sync_all();
    if (warp == 2) { tc_fence_after(); xtmem_dealloc<2>(tmem_base, 512); }
}

}  // namespace

extern "C" {


cudaError_t omni_attn_configure(void) {
    return cudaFuncSetAttribute(attention_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_SMEM_BYTES);
}

cudaError_t omni_launch_rope_freq(double theta, double *freq, cudaStream_t s) {
    rope_freq_kernel<<<1, HD / 2, 0, s>>>(theta, freq);
    return cudaGetLastError();
}

cudaError_t omni_launch_attn_prep(const void *qkv, const float *qw, const float *kw, const int32_t *pos, const double *freq,
                                  const int32_t *vcol, int T, int head_stride, int vpitch, float eps, void *Q, void *K, void *Vt,
                                  uint32_t *status, cudaStream_t s) {
    const int tokens = PREP_THREADS / 32 / PREP_WARPS, prep = (T + tokens - 1) / tokens;
    return omni_launch_chain(attn_prep_kernel, dim3(prep + (T + 63) / 64 * OMNI_NKV), dim3(PREP_THREADS), 0, s,
                             (const __nv_bfloat16 *)qkv, qw, kw, pos, freq, vcol, T, prep, head_stride, vpitch, eps, (__nv_bfloat16 *)Q,
                             (__nv_bfloat16 *)K, (__nv_bfloat16 *)Vt, status);
}

// tiles: [n_tiles] of {record start, first query row, rows (<= 128), Vt column of the record start}
cudaError_t omni_launch_attention(const CUtensorMap *tm_q, const CUtensorMap *tm_k, const CUtensorMap *tm_vt, const void *tiles,
                                  int n_tiles, int T, void *out, uint32_t *status, int early_dependents, int n_sm, cudaStream_t s) {
    const int n_items = n_tiles * AT_PAIRS_PER_TILE, pairs = n_items < n_sm / 2 ? n_items : n_sm / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(AT_THREADS);
    cfg.dynamicSmemBytes = AT_SMEM_BYTES;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = omni_dependent_launch_enabled() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, attention_kernel, *tm_q, *tm_k, *tm_vt, (const AttnTile *)tiles, n_items, T, 1.0f / sqrtf((float)OMNI_HD),
                              (__nv_bfloat16 *)out, early_dependents, status);
}

}  // extern "C"
