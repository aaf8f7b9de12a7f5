// The two dense projections of the attention half for short batches (sm_100a).
//
// On CTA pairs (expert_pair_kernel) a batch of one token tile gives the q|k|v projection 20 items of 256 weight
// rows and the output projection 8: 40 and 16 of 148 SMs stream 21 and 17 MB of weights, 11.5 and 16.5 us
// where the memory would need 3.  Here a CTA takes 40 (16) weight rows and all token rows: 128 CTAs for
// either projection.  What a CTA pays for that is the token operand, which every CTA reads whole
// through its SM (1 MB at 128 rows of 4096), so longer batches stay on the pairs.  Attention half on pairs and here, both in
// turn: 1 token 41.4 -> 27.0 us, 37 44.5 -> 29.2, 100 45.3 -> 34.8, 128 46.0 -> 37.1; the line lies at the longest token operand of one
// CTA here, not where the two would be equal.
//
// The weight rows are the first rows of an M = 128 operand (M = 64 for the output projection: 256 instructions of K = 16 read half as
// much of shared memory, attention half of 37 tokens 31.0 -> 28.9 us, 128 38.0 -> 36.8); its other rows are whatever follows in shared memory
// and feed accumulator lanes that are never read.  K runs in the order of the pair kernel and into one
// accumulator, so the results are its bits.  Every wait is bounded.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "omni_internal.h"
#include "omni_pair.cuh"
#include "omni_pdl.cuh"
#include "omni_ptx.cuh"

namespace {

enum { THIN_QKV = 0, THIN_OPROJ = 1 };
template <int MODE> struct ThinCfg;
template <> struct ThinCfg<THIN_QKV> { static constexpr int ROWS = OMNI_THIN_QKV_ROWS, MMA_ROWS = 128, K = OMNI_H, COLS = OMNI_QKV; };
template <> struct ThinCfg<THIN_OPROJ> { static constexpr int ROWS = OMNI_THIN_OPROJ_ROWS, MMA_ROWS = 64, K = OMNI_NH * OMNI_HD, COLS = OMNI_H; };

constexpr int TN_THREADS = 256;          // warp 0 and 4 epilogue of accumulator lanes 0..31 (half of the tokens each), 1 MMA, 2 TMEM, 3 TMA, 5 epilogue of lanes 32..
constexpr int TN_MAX_STAGES = 12, TN_RING_BYTES = 200 * 1024;
constexpr int TN_SMEM_BYTES = TN_RING_BYTES + A_TILE_BYTES + 1024 + 8 * (2 * TN_MAX_STAGES + 1) + 16 + 4 * TN_MAX_STAGES;   // the operand of the last slab reads 128 rows
static_assert(TN_SMEM_BYTES <= 232448, "shared memory budget");

__device__ __forceinline__ void tma_load_3d_hint(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5}], [%2], %6;"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z), "l"(policy) : "memory");
}

template <int MODE>
__global__ void __launch_bounds__(TN_THREADS, 1)
dense_thin_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, int T, int n, int stages,
                  __nv_bfloat16 *__restrict__ out, float *__restrict__ resid, uint32_t *__restrict__ status) {
    using C = ThinCfg<MODE>;
    constexpr int STEPS = C::K / (BK * OMNI_THIN_SLABS), W_SLAB = C::ROWS * BK * 2;
    const int x_slab = n * BK * 2, stage_bytes = OMNI_THIN_SLABS * (W_SLAB + x_slab);
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *const smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar_base = smem_base + TN_RING_BYTES + A_TILE_BYTES;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (TN_MAX_STAGES + s); };
    const uint32_t done_bar = bar_base + 8u * (2 * TN_MAX_STAGES);
    uint8_t *misc = smem_gen + TN_RING_BYTES + A_TILE_BYTES + 8 * (2 * TN_MAX_STAGES + 1);
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(misc);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(misc + 4);
    volatile int *armed = reinterpret_cast<volatile int *>(misc + 16);
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int col0 = blockIdx.x * C::ROWS;
    const Abort ab{abort_flag, 0u, status};

    if (threadIdx.x == 0) {
        for (int s = 0; s < TN_MAX_STAGES; s++) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); armed[s] = -1; }
        mbar_init(done_bar, 1);
        *abort_flag = 0;
        fence_mbar_init();
        prefetch_tmap(&tm_w);
        prefetch_tmap(&tm_x);
    }
    if (warp == 2) { tmem_alloc(smem_u32((const void *)tmem_slot), 128); tmem_relinquish(); }
    dep_wait();
    dep_launch();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 3 && elect_one()) {
        PipeState p;
        const uint64_t pol_w = l2_policy_evict_first(), pol_x = l2_policy_evict_last();
        for (int ks = 0; ks < STEPS; ks++) {
            if (!mbar_wait(empty_bar(p.stage), p.phase ^ 1u, abort_flag, status)) break;
            const uint32_t st = smem_base + p.stage * stage_bytes;
            armed[p.stage] = (int)p.phase;
            mbar_expect_tx(full_bar(p.stage), (uint32_t)stage_bytes);
            tma_load_3d_hint(st, &tm_w, 0, col0, ks * OMNI_THIN_SLABS, full_bar(p.stage), pol_w);
            tma_load_3d_hint(st + OMNI_THIN_SLABS * W_SLAB, &tm_x, 0, 0, ks * OMNI_THIN_SLABS, full_bar(p.stage), pol_x);
            p.advance(stages);
        }
    } else if (warp == 1 && elect_one()) {
        PipeState p;
        const uint32_t idesc = idesc_bf16(C::MMA_ROWS, n);
        for (int ks = 0; ks < STEPS; ks++) {
            if (!mbar_wait(full_bar(p.stage), p.phase, abort_flag, status)) break;
            tc_fence_after();
            const uint32_t st = smem_base + p.stage * stage_bytes;
#pragma unroll
            for (int s = 0; s < OMNI_THIN_SLABS; s++) {
                const uint64_t da = smem_desc_sw128(st + s * W_SLAB), db = smem_desc_sw128(st + OMNI_THIN_SLABS * W_SLAB + s * x_slab);
#pragma unroll
                for (int k = 0; k < BK / 16; k++) umma_bf16(tmem_base, da + 2u * k, db + 2u * k, idesc, (ks | s | k) ? 1u : 0u);
            }
            umma_commit(empty_bar(p.stage));
            p.advance(stages);
        }
        umma_commit(done_bar);
    } else if (warp == 0 || warp == 4 || (warp == 5 && C::ROWS > 32)) {
        const int q = warp & 3, row = q * 32 + lane;                          // accumulator lane = weight row of this CTA
        const bool mine = row < C::ROWS;
        const int chunks = (T + 31) >> 5;
        const int c0 = warp == 4 ? (chunks + 1) >> 1 : 0, c1 = warp == 0 ? (chunks + 1) >> 1 : chunks;
        const uint32_t t0 = tmem_base + ((uint32_t)(q * 32) << 16);
        if constexpr (MODE == THIN_OPROJ) {
            // the residual is loaded while the product runs
            float old[2][32];
            float *xr = resid + col0 + row;
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const int t = (c0 + i) * 32 + j;
                    old[i][j] = mine && c0 + i < c1 && t < T ? xr[(long)t * C::COLS] : 0.f;
                }
            if (xwait_warp<false>(done_bar, 0, ab)) {
                tc_fence_after();
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    if (c0 + i < c1) {
                        uint32_t v[32];
                        tmem_ld32(t0 + (c0 + i) * 32, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; j++) {
                            const int t = (c0 + i) * 32 + j;
                            if (mine && t < T) xr[(long)t * C::COLS] = old[i][j] + __uint_as_float(v[j]);
                        }
                    }
                }
            }
        } else if (xwait_warp<false>(done_bar, 0, ab)) {
            tc_fence_after();
            for (int c = c0; c < c1; c++) {
                uint32_t v[32];
                tmem_ld32(t0 + c * 32, v);
                tmem_ld_wait();
                __nv_bfloat16 *o = out + (long)c * 32 * C::COLS + col0 + row;
#pragma unroll
                for (int j = 0; j < 32; j++)
                    if (mine && c * 32 + j < T) o[(long)j * C::COLS] = __float2bfloat16_rn(__uint_as_float(v[j]));
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0) {
        // a wait ran out: give loads in flight, and the MMAs that may still be reading them, a bounded chance to finish
        for (int s = 0; s <= stages; s++) {
            const int par = s < stages ? armed[s] : 0;
            if (par < 0) continue;
            const uint64_t t1 = globaltimer_ns();
            while (!mbar_try_wait(s < stages ? full_bar(s) : done_bar, (uint32_t)par) && globaltimer_ns() - t1 < 50000000ull) {}
        }
    }
    __syncthreads();
    if (warp == 2) { tc_fence_after(); tmem_dealloc(tmem_base, 128); }
}

template <int MODE>
cudaError_t launch_thin(const CUtensorMap *tm_w, const CUtensorMap *tm_x, int T, void *out, float *resid, uint32_t *status, cudaStream_t s) {
    using C = ThinCfg<MODE>;
    static_assert(C::COLS % C::ROWS == 0 && C::ROWS % 8 == 0, "weight rows per CTA");
    const int n = (T + 15) & ~15, stage = OMNI_THIN_SLABS * (C::ROWS + n) * BK * 2, fit = TN_RING_BYTES / stage;
    return omni_launch_chain(dense_thin_kernel<MODE>, dim3(C::COLS / C::ROWS), dim3(TN_THREADS), TN_SMEM_BYTES, s, *tm_w, tm_x[n / 16 - 1], T, n,
                             fit < TN_MAX_STAGES ? fit : TN_MAX_STAGES, (__nv_bfloat16 *)out, resid, status);
}

}  // namespace

extern "C" {

cudaError_t omni_dense_configure(void) {
    cudaError_t e = cudaFuncSetAttribute(dense_thin_kernel<THIN_QKV>, cudaFuncAttributeMaxDynamicSharedMemorySize, TN_SMEM_BYTES);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(dense_thin_kernel<THIN_OPROJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, TN_SMEM_BYTES);
}

cudaError_t omni_launch_dense_thin(int which, const CUtensorMap *tm_w, const CUtensorMap *tm_x, int T, void *out_bf16, float *resid,
                                   uint32_t *status, cudaStream_t s) {
    if (T <= 0 || T > OMNI_THIN_MAX_ROWS) return cudaErrorInvalidValue;
    return which == 0 ? launch_thin<THIN_QKV>(tm_w, tm_x, T, out_bf16, resid, status, s)
                      : launch_thin<THIN_OPROJ>(tm_w, tm_x, T, out_bf16, resid, status, s);
}

}  // extern "C"
