// The two grouped expert products of the Clef-Omni MoE block on pairs of SMs (sm_100a):
//   expert_pair_kernel<GATEUP>  per expert: h = silu(Xe Wg^T) * (Xe Wu^T), SwiGLU in the epilogue
//                               (reference: metal/clef.metal:2455-2492, omni_expert_gemm + omni_swiglu;
//                               on one GPU the token rows are fetched through the permutation
//                               here: metal/clef.metal:2445-2453, omni_gather)
//   expert_pair_kernel<DOWN>    per expert: d = He Wd^T            (clef.metal:2455-2482)
//
// Two CTAs of a cluster (two SMs) work on one item together: one tcgen05.mma.cta_group::2 of
// shape M = 256 weight rows x N <= 256 token rows.  Each CTA loads its own 128 weight rows and
// HALF of the token rows into its own shared memory (plain per-CTA TMA loads or 16-byte
// cp.async gathers); the tensor cores of the two SMs exchange the token halves themselves, so a
// token row crosses the L2 -> SM path once per 256 weight rows instead of once per 128.  Each
// CTA ends up with the accumulator of its own 128 weight rows (128 lanes x N columns of its
// tensor memory), twice buffered, so the epilogue of one item runs under the MMAs of the next.
//
// Gate/up: the 128 weight rows of a CTA are 64 gate rows and the 64 up rows of the same
// intermediate columns, interleaved in blocks of 16 by a four-dimensional TMA box over the
// [gate rows; up rows] matrix of the expert.  Gate and up of one column are then 16 lanes apart in
// one accumulator and reach the same thread's registers in the two 16-lane loads of a quadrant:
// SwiGLU needs neither a lane exchange nor a second accumulator.
//
// Epilogue: TMEM -> registers in the layout of an 8x8 matrix fragment (tcgen05.ld.16x256b) ->
// stmatrix.trans into a row-major tile in shared memory (four 16-byte rows per lane group instead
// of one 2-byte store per element) -> whole 128- or 256-byte row pieces written with 16-byte stores.  With expert parallelism the down product writes each
// row piece straight into the buffer of the rank that owns the token (plain peer stores), so
// the way back travels under the product, tile by tile, and no separate copy kernel runs.
//
// The same code runs with CTAS = 1 (no cluster, tcgen05 cta_group::1).  No load anywhere uses
// the cluster-multicast form.  Every wait is bounded; when one runs out the CTA (and its peer)
// raise OMNI_ST_TIMEOUT, drain what they issued, free tensor memory and return.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

#include "omni_internal.h"
#include "omni_ep_dev.cuh"
#include "omni_land.cuh"
#include "omni_meet.cuh"
#include "omni_pair.cuh"
#include "omni_pdl.cuh"
#include "omni_ptx.cuh"

namespace {

__device__ __forceinline__ void named_bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// 16 TMEM lanes x 32 columns: register 4i + {0,1} of lane t holds row t/4, columns 8i + 2(t%4) + {0,1},
// register 4i + {2,3} row t/4 + 8 of the same columns.
__device__ __forceinline__ void tmem_ld_16x32(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}
// four 8x8 matrices, transposed: lane i supplies the address of one 16-byte row
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// ------------------------------------------------------------------ configuration
enum { X_GATEUP = 0, X_DOWN = 1,
       // the two dense projections of the attention half, run as "one expert" over all token rows:
       X_QKV = 2,      // P[T][5120] = xn[T][2048] . W_qkv^T, BF16 out
       X_OPROJ = 3 };  // x[T][2048] += A[T][4096] . W_out^T, added into the FP32 residual

// ROWS: accumulator rows (weight rows) of one CTA; OUTC: output columns one CTA produces;
// MT: such CTA-level weight tiles per expert.
template <int MODE> struct XMode;
template <> struct XMode<X_GATEUP> { static constexpr int KTOT = OMNI_H, OUTC = 64, MT = OMNI_F / 64, OUT_COLS = OMNI_F; };
template <> struct XMode<X_DOWN> { static constexpr int KTOT = OMNI_F, OUTC = 128, MT = OMNI_H / 128, OUT_COLS = OMNI_H; };
template <> struct XMode<X_QKV> { static constexpr int KTOT = OMNI_H, OUTC = 128, MT = OMNI_QKV / 128, OUT_COLS = OMNI_QKV; };
template <> struct XMode<X_OPROJ> { static constexpr int KTOT = OMNI_NH * OMNI_HD, OUTC = 128, MT = OMNI_H / 128, OUT_COLS = OMNI_H; };

template <int MODE, int CTAS> struct XCfg {
    using M = XMode<MODE>;
    static constexpr int TOK_ROWS = 128;                                // token rows one CTA stages per K slab: all of a tile, or half
    static constexpr int T_BYTES = TOK_ROWS * BK * 2;                   // 16 KiB
    static constexpr int W_BYTES = A_TILE_BYTES;                        // 16 KiB: 128 weight rows
    // the epilogue stages 32 token rows at a time, twice buffered, per half of its warps; the
    // output projection stores from registers
    static constexpr int CHUNK_BYTES = 32 * M::OUTC * 2;
    static constexpr int STAGE_OUT_BYTES = MODE == X_OPROJ ? 0 : 4 * CHUNK_BYTES;   // 16 KiB (gate/up) or 32 KiB
    // Ring depths (stages of 64 K elements).  A slab lasts 512 clocks at 256 token rows and a load takes
    // 1500 to 2500 under load, so everything that is not needed elsewhere goes into the rings: with
    // a whole 64 KiB output tile in shared memory and 4 token stages the dense projections
    // waited for tokens half of the time (847 clocks per slab).
    static constexpr int STAGES = MODE == X_OPROJ ? 7 : 6;
    static constexpr int RING_BYTES = STAGES * (W_BYTES + T_BYTES);
    static constexpr int TOTAL_BYTES = RING_BYTES + STAGE_OUT_BYTES + 1024 + 1024;
    static constexpr int ITEMS_PER_TILE = M::MT / CTAS;
};
static_assert(XCfg<X_QKV, 2>::TOTAL_BYTES <= 232448 && XCfg<X_OPROJ, 2>::TOTAL_BYTES <= 232448 &&
              XCfg<X_GATEUP, 1>::TOTAL_BYTES <= 232448 && XCfg<X_DOWN, 1>::TOTAL_BYTES <= 232448 &&
              XCfg<X_GATEUP, 2>::TOTAL_BYTES <= 232448 && XCfg<X_DOWN, 2>::TOTAL_BYTES <= 232448, "shared memory budget");

constexpr int X_THREADS = 384;      // warp 0 weight loads, 1 MMA, 2 TMEM + scheduler, 3 token loads, 4..11 epilogue
constexpr int X_GATHER_THREADS = 128;   // gate/up only: warps 12..15 fetch the token rows through the permutation
constexpr int X_COPY_THREADS = 128; // with COPY: warps 16..19 move this rank's token rows to the other ranks
constexpr int X_EPI_WARPS = 8;
template <int MODE, bool COPY> constexpr int x_threads() { return X_THREADS + (MODE == X_GATEUP ? X_GATHER_THREADS : 0) + (COPY ? X_COPY_THREADS : 0); }
constexpr int X_RING = 4;
constexpr int X_MAX_STAGES = 8;     // of the rings; 64 bytes of announced parities

struct XArgs {
    const omni_ttile *ttiles;
    const int32_t *n_ttiles;
    int32_t *work_counter;
    __nv_bfloat16 *out;                 // h [rows][768], d [rows][2048] or the q|k|v projections [rows][5120]
    float *resid;                       // output projection: the FP32 residual stream it adds into
    uint32_t *status;
    // expert parallelism, overlap mode: rows of a group of experts may be read once ready[grp] == need[grp]
    const uint32_t *ready;
    const int32_t *need;
    int group_size;
    // gate/up on one GPU: token row i of the permuted order is row gather_rows[i] of gather_src
    const __nv_bfloat16 *gather_src;
    const int32_t *gather_rows;
    // expert parallelism (pe.world > 1).  Down: result row i goes to row (rowinfo[i] & 0xfffff) of
    // pe.dret[rowinfo[i] >> 20], the buffer of the rank the token came from.  Gate/up with copy
    // warps: the spare warps send this rank's token rows (row rowmap[r] of disp_src for permuted
    // row r) to the owners of their experts while the other warps compute.
    omni_ep_peers pe;
    const int32_t *rowinfo;
    omni_ep_send send;                  // what the copy warps send from
    int need_blocks;                    // > 0: an arrival counter is complete at this value (it counts sender blocks), else at need[group]
    int early_dependents;
    const char *weights;                // down on one GPU: the matrix behind tm_w, for prefetches
    int dense_rows, dense_tiles;        // dense projections: token rows, and the near-equal tiles they are cut into
};

constexpr int DENSE_MIN = 96, DENSE_ITEM = 56;    // of the choice of tile length in omni_launch_dense_pair, in rows
constexpr int DENSE_GROUP = 16;     // token tiles (of up to 256 rows, 1 to 2 MiB) that share a sweep over the weight blocks of a dense projection
struct WorkSlotX { int expert, row0, len, m; };

// silu(g) * u with silu(g) = g * sigmoid(g) = (g/2) * (1 + tanh(g/2)): one special-function
// instruction per element instead of two (exp and reciprocal).  tanh.approx.f32 is accurate to
// about 2^-11 absolute; the result is rounded to BF16 (2^-9 relative) right after.
__device__ __forceinline__ float silu_mul(float g, float u) {
    const float hg = 0.5f * g;
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(hg));
    return fmaf(hg, t, hg) * u;
}

// ====================================================================== the kernel
// Work distribution: an expert-major list of token tiles, items
// (token tile, weight block) claimed one at a time from a device counter by the first CTA of the
// pair, which hands each decoded item to the consumers of BOTH CTAs through a small ring that
// exists in each CTA's shared memory.
template <int MODE, int CTAS, bool COPY>
__global__ void __launch_bounds__((x_threads<MODE, COPY>()), 1)
expert_pair_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ TokMaps tm_tok, const __grid_constant__ XArgs a) {
    using C = XCfg<MODE, CTAS>;
    using M = XMode<MODE>;
    constexpr int KSTAGES = M::KTOT / BK;
    constexpr int STAGES = C::STAGES, MI = C::ITEMS_PER_TILE;
    constexpr bool PAIR = CTAS == 2;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *const smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t tok_base = smem_base + STAGES * C::W_BYTES;
    uint8_t *const out_tile = smem_gen + C::RING_BYTES; // 4 x [32][OUTC] bf16: two chunks per epilogue half, none for the output projection
    const uint32_t bar_base = smem_base + C::RING_BYTES + C::STAGE_OUT_BYTES;
    // A stage of weights and one of tokens share their two barriers, so that the MMA warp waits and commits
    // once per slab.  Its loop costs about 400 clocks per slab with two waits (70 to 90 each, also when the phase is complete) and two
    // commits, more than the MMAs of a tile of up to ~190 rows.  us, two rings of barriers -> one, in turn, each alone under its own
    // clock, on two GPUs: block of 9 tokens 97.5 -> 96.3 and 98.6 -> 97.4, 128 and 1030 the same, 2048 273.3 -> 270.4 and 283.4 -> 282.7, 4096
    // 416.8 -> 406.4 and 445 -> 436, 8192 715 -> 701 and 770 -> 759, 16384 1301 -> 1296 and 1368 -> 1354; attention half of 37 tokens the same, 129
    // 46.6 -> 43.3 and 45.8 -> 43.7, 300 48.4 -> 45.3 and 47.6 -> 45.3, 700 57.2 -> 54.5 and 56.4 -> 54.4, 1030 in 6 records 64.7 -> 63.0 and 64.6 -> 62.7,
    // 4096 in 8 204.8 -> 202.9 and the same.
    // On single CTAs nine (gate/up) and eight (down) stages of weights and four of tokens became six of both.  A layer whose experts stay in
    // L2, and 16 layers in turn (1.2 GB of touched experts, from memory): 1 token 35.4 -> 33.3 and 35.8 -> 34.1, 2 tokens 47.2 -> 46.7 and
    // 49.9 -> 48.8; longer batches on single CTAs, 9 tokens 111.7 -> 106.6, 128 200.1 -> 199.6, 1030 246 -> 238, 4096 578 -> 548.
    // (Two slabs per turn of the loop, or a look at the next slab's barrier ahead of the MMAs: up to 2 % slower, and no change.)
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
    auto afull_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + b); };
    auto aempty_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + 2 + b); };
    const uint32_t drain_bar = bar_base + 8u * (2 * STAGES + 4);
    auto ifull_bar = [&](int r) { return bar_base + 8u * (2 * STAGES + 5 + r); };
    auto iempty_bar = [&](int r) { return bar_base + 8u * (2 * STAGES + 5 + X_RING + r); };
    constexpr int N_BARS = 2 * STAGES + 5 + 2 * X_RING;
    constexpr int MISC_OFF = (N_BARS * 8 + 15) & ~15;            // the item ring is written with 16-byte stores
    constexpr int RING_OFF = 16 + 2 * X_MAX_STAGES * 4;
    static_assert(STAGES <= X_MAX_STAGES && RING_OFF % 16 == 0 && MISC_OFF + RING_OFF + X_RING * 16 <= 1024, "barrier block");
    uint8_t *misc = smem_gen + C::RING_BYTES + C::STAGE_OUT_BYTES + MISC_OFF;
    const uint32_t misc_u32 = bar_base + MISC_OFF;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(misc);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(misc + 4);
    volatile short *epi_quit = reinterpret_cast<volatile short *>(misc + 8);    // [half][item parity] a warp of this epilogue half gave up
    volatile int *armed_w = reinterpret_cast<volatile int *>(misc + 16);        // [STAGES] parity with which weights were announced last, -1 none
    volatile int *armed_t = armed_w + STAGES;                                   // [STAGES] the same for tokens that come by TMA
    volatile WorkSlotX *ring = reinterpret_cast<volatile WorkSlotX *>(misc + RING_OFF);
    const uint32_t ring_u32 = misc_u32 + RING_OFF;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? __shfl_sync(0xffffffffu, cluster_ctarank(), 0) : 0u;      // uniform for the compiler, like the warp index
    const bool leader = rank == 0;
    const bool gathering = a.gather_src != nullptr;
    const Abort ab{abort_flag, PAIR ? mapa_u32(misc_u32 + 4, rank ^ 1u) : 0u, a.status};
    // a barrier of the pair's first CTA, as an address every CTA of the pair may signal
    auto lead = [&](uint32_t bar) { return PAIR ? mapa_u32(bar, 0) : bar; };
    auto arrive_lead = [&](uint32_t bar) { if (PAIR) mbar_arrive_remote(mapa_u32(bar, 0)); else mbar_arrive(bar); };

    if (threadIdx.x == 0) {
        const int tp = gathering ? X_GATHER_THREADS / 32 : 1;                       // arrivals of a CTA's token producer per item
        const int tok_arrivals = gathering ? X_GATHER_THREADS * CTAS : 1;
        for (int s = 0; s < STAGES; s++) { mbar_init(full_bar(s), 1 + tok_arrivals); mbar_init(empty_bar(s), 1); }
        for (int s = 0; s < 2 * STAGES; s++) armed_w[s] = -1;
        for (int b = 0; b < 2; b++) { mbar_init(afull_bar(b), 1); mbar_init(aempty_bar(b), X_EPI_WARPS * CTAS); }
        mbar_init(drain_bar, 1);
        // consumers of an item: in either CTA the weight producer, the token producer(s) and the epilogue
        // warps; in the first also the MMA thread
        for (int r = 0; r < X_RING; r++) {
            mbar_init(ifull_bar(r), 1);
            mbar_init(iempty_bar(r), 1 + CTAS * (1 + tp + X_EPI_WARPS));
        }
        *abort_flag = 0;
        for (int i = 0; i < 4; i++) epi_quit[i] = 0;
        fence_mbar_init();
        prefetch_tmap(&tm_w);
        for (int i = 0; i < OMNI_TOK_BOXES; i++) prefetch_tmap(&tm_tok.m[i]);
    }
    // the peer's barriers must exist before anything of this CTA can signal them
    if (PAIR) cluster_sync_all(); else __syncthreads();
    if (warp == 2) xtmem_alloc<CTAS>(smem_u32((const void *)tmem_slot), 512);
    if (MODE == X_DOWN && a.weights && warp == 3 && lane < 128 * M::KTOT * 2 / OMNI_PREFETCH_PIECE) {
        // CTAs become resident one after the other while the last items of gate/up leave memory half idle: each asks for the
        // weights of its first item, one contiguous piece, to be brought into L2 (us per block, both in turn: 1 token 36.7 -> 35.3, 3 55.6 ->
        // 54.5, 9 108.4 -> 103.5, 37 183.4 -> 180.6, 128 202.1 -> 200.8, 511 and 1030 the same, 2048 284.0 -> 281.6).  The tile list is older than
        // the kernel in front (omni_pdl.cuh); whatever it held, the address stays inside the matrix.
        const int w0 = (int)blockIdx.x / CTAS;
        const int4 t = __ldcg(reinterpret_cast<const int4 *>(a.ttiles) + w0 / MI);
        const int cnt = max(t.w >> 16, 1), m = ((w0 - (t.w & 0xffff) * MI) / cnt) & (MI - 1);
        const char *p = a.weights + ((size_t)(t.x & (OMNI_E - 1)) * M::OUT_COLS + (m * CTAS + rank) * 128) * (M::KTOT * 2) + lane * OMNI_PREFETCH_PIECE;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(OMNI_PREFETCH_PIECE) : "memory");
    }
    dep_wait();                 // everything above overlaps the tail of the previous kernel
    if (a.early_dependents) dep_launch();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = (uint32_t)uniform_i32((int)*tmem_slot);

    // weight tile of CTA `rank` for block m of an expert, K slab ks
    auto load_weights = [&](uint32_t dst, int expert, int m, int ks, uint32_t bar, uint64_t pol) {
        const int m_cta = m * CTAS + (int)rank;
        if (MODE == X_GATEUP) xtma_4d<CTAS>(dst, &tm_w, ks * BK, 0, 0, expert * (2 * OMNI_F / 16) + m_cta * 4, bar, pol);
        else xtma_2d<CTAS>(dst, &tm_w, ks * BK, expert * M::OUT_COLS + m_cta * 128, bar, pol);
    };

    if (warp == 2 && leader && elect_one()) {
        // ---------------------------------------------------------- scheduler
        // Claims items and hands them, decoded, to the consumers of both CTAs.  Its own warp: an item
        // costs an atomic, up to two dependent global loads and a cluster-scope release (about 2 us), which
        // inside the weight producer's loop held up the loads of every item (12 slabs of 512 clocks in
        // the down product).  The claim of the item after the next is in flight meanwhile.  The first item needs
        // no claim (the counter hands out those behind one per pair), and its tile is loaded beside the length of the list.
        constexpr bool DENSE = MODE == X_QKV || MODE == X_OPROJ;
        PipeState wr;
        auto tile_at = [&](int i) {
            const int4 v = __ldcg(reinterpret_cast<const int4 *>(a.ttiles) + i);
            return omni_ttile{v.x, v.y, v.z, v.w};
        };
        const int n_pairs = (int)gridDim.x / CTAS;
        int w0 = (int)blockIdx.x / CTAS;
        omni_ttile head = omni_ttile{0, 0, 0, 0};
        if (!DENSE) head = tile_at(w0 / MI);                  // below OMNI_MAX_TTILES for any grid; only used if the list is that long
        const int n_work = (DENSE ? a.dense_tiles : __ldcg(a.n_ttiles)) * MI;
        for (bool first_item = true;; first_item = false) {
            const int w1 = DENSE ? w0 + n_pairs : n_pairs + atomicAdd(a.work_counter, 1);
            int m = 0;
            omni_ttile cur = omni_ttile{0, 0, -1, 0};
            if (DENSE && w0 < n_work) {
                // equal items, dealt out in turn: the weight blocks of a group of token tiles before the next
                // group, so that the token rows in use stay in L2
                const int group = w0 / (DENSE_GROUP * MI), first = group * DENSE_GROUP;
                const int cnt = min(DENSE_GROUP, a.dense_tiles - first), local = w0 - first * MI;
                m = local / cnt;
                const int t = first + local % cnt, base = a.dense_rows / a.dense_tiles, extra = a.dense_rows % a.dense_tiles;
                cur = omni_ttile{0, t * base + min(t, extra), base + (t < extra), 0};
            } else if (w0 < n_work) {                         // item -> (weight block m, tile of the expert)
                if (!first_item) head = tile_at(w0 / MI);
                const int first = head.group & 0xffff, cnt = head.group >> 16, local = w0 - first * MI;
                m = local / cnt;
                const int at = first + local % cnt;
                cur = at == w0 / MI ? head : tile_at(at);
            }
            if (!xwait_lazy(iempty_bar(wr.stage), wr.phase ^ 1u, ab)) break;
            ring[wr.stage].expert = cur.expert; ring[wr.stage].row0 = cur.row0;
            ring[wr.stage].len = cur.len; ring[wr.stage].m = m;
            mbar_arrive(ifull_bar(wr.stage));
            if (PAIR) {
                st_cluster_v4(mapa_u32(ring_u32 + 16u * wr.stage, 1), cur.expert, cur.row0, cur.len, m);
                mbar_arrive_cluster(mapa_u32(ifull_bar(wr.stage), 1));
            }
            if (cur.len < 0) break;                           // told the consumers to stop
            wr.advance(X_RING);
            w0 = w1;
        }
    } else if (warp == 0) {
        // ---------------------------------------------------------- weight producer (of each CTA)
        // This warp, the token producer's and the MMA issuer's run their loops with all lanes
        // together and elect a thread only to issue.  With the loop inside the elected branch it
        // depended on the instantiation whether the compiler kept stages and descriptors in
        // uniform registers; where it did not, a slab took 770 clocks to issue instead of 512.
        PipeState p, wr;
        // evict first even when the expert has further token tiles: neighbouring pairs read those at the
        // same time and meet in L2 all the same (kept with evict_last the weights displaced the
        // token rows and the results: gate/up at 4096 tokens 190 us, now 179)
        const uint64_t pol_w = l2_policy_evict_first();
        bool ok = true;
        while (ok) {
            ok = xwait_warp<PAIR>(ifull_bar(wr.stage), wr.phase, ab);
            if (!ok) break;
            const int expert = uniform_i32(ring[wr.stage].expert), len = uniform_i32(ring[wr.stage].len), m = uniform_i32(ring[wr.stage].m);
            if (elect_one()) arrive_lead(iempty_bar(wr.stage));
            wr.advance(X_RING);
            if (len < 0) break;
            for (int ks = 0; ks < KSTAGES; ks++) {
                ok = xwait_warp<false>(empty_bar(p.stage), p.phase ^ 1u, ab);
                if (!ok) break;
                if (elect_one()) {
                    if (leader) {
                        armed_w[p.stage] = (int)p.phase;
                        mbar_expect_tx(full_bar(p.stage), CTAS * C::W_BYTES);       // this CTA's tile and the peer's
                    }
                    load_weights(smem_base + p.stage * C::W_BYTES, expert, m, ks, lead(full_bar(p.stage)), pol_w);
                }
                p.advance(STAGES);
            }
        }
    } else if (MODE == X_GATEUP && gathering && warp >= 12 && warp < 16) {
        // ---------------------------------------------------------- token producer, gathering
        // 128 threads fetch this CTA's share of the tile's token rows through the permutation:
        // 16-byte asynchronous copies, eight threads per 128-byte row segment, stored in the
        // 128-byte-swizzled layout the MMA descriptors expect (chunk c of row r at c ^ (r & 7)
        // inside its 8-row group).  A stage is handed to the MMA thread LAG stages after it was
        // issued, once the copies have landed and are ordered before the tensor core's reads.
        constexpr int LAG = CTAS == 2 ? 3 : 2;
        static_assert(STAGES > LAG, "token ring too short for the copy lag");
        constexpr int RSTEP = X_GATHER_THREADS / 8, NR = C::TOK_ROWS / RSTEP;
        const uint64_t pol_t = l2_policy_evict_last();
        const int gt = threadIdx.x - X_THREADS;
        const int c = gt & 7, rb = gt >> 3;                           // chunk of the row segment; first of this thread's rows
        const uint32_t dst_off = (uint32_t)(rb * 128 + ((c ^ (rb & 7)) << 4));
        const char *src0 = reinterpret_cast<const char *>(a.gather_src) + c * 16;
        PipeState p, pend, wr;
        int off[NR], off_next[NR];
        int ready_group = -1;
        auto next_item = [&](int (&o)[NR]) -> int {
            if (!xwait_warp<PAIR>(ifull_bar(wr.stage), wr.phase, ab)) return -1;
            const int row0 = ring[wr.stage].row0, len = ring[wr.stage].len, expert = ring[wr.stage].expert;
            __syncwarp();
            if (lane == 0) arrive_lead(iempty_bar(wr.stage));
            wr.advance(X_RING);
            if (a.ready && len >= 0) {
                // expert parallelism: the rows and the row map of this expert's group are written by
                // other GPUs while the kernel runs; they are complete once the arrival counters of
                // every group up to it are (a token row may have come with an earlier group)
                const int grp = expert / a.group_size;
                bool ok = true;
                while (ready_group < grp && ok) {
                    const int g2 = ready_group + 1;
                    if (lane == 0) {
                        const uint32_t want = a.need_blocks ? (uint32_t)a.need_blocks : (uint32_t)a.need[g2];
                        const uint64_t t0 = globaltimer_ns();
                        while (ld_acquire_sys_u32(a.ready + g2) != want) {
                            __nanosleep(200);
                            if (*abort_flag || globaltimer_ns() - t0 > WAIT_LIMIT_NS) {
                                ab.raise(OMNI_ST_TIMEOUT | OMNI_ST_TIMEOUT_ARRIVAL);
                                ok = false;
                                break;
                            }
                        }
                    }
                    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                    ready_group = g2;
                }
                if (!ok) return -1;
            }
            const int share = (((len + 15) & ~15) / CTAS);            // token rows of the tile each CTA stages
            const int first = (int)rank * share;
#pragma unroll
            for (int i = 0; i < NR; i++) {
                const int r = rb + RSTEP * i;
                o[i] = (r < share && first + r < len) ? __ldcv(a.gather_rows + row0 + first + r) * (OMNI_H * 2) : -1;
            }
            return len;
        };
        // hands the oldest stage still in flight to the MMA thread once at most `left` newer ones are
        auto hand_over = [&](auto left) {
            cp_async_wait<decltype(left)::value>();
            fence_proxy_async_smem();
            arrive_lead(full_bar(pend.stage));
            pend.advance(STAGES);
        };
        int len = next_item(off);
        while (len >= 0) {
            bool ok = true;
            for (int ks = 0; ks < KSTAGES; ks++) {
                // hand over before blocking on a free stage: the MMA thread must never wait for
                // this loop to issue further copies
                if (ks >= LAG) hand_over(std::integral_constant<int, LAG - 1>{});
                ok = xwait_warp<false>(empty_bar(p.stage), p.phase ^ 1u, ab);
                if (!ok) break;
                const uint32_t sb = tok_base + p.stage * C::T_BYTES + dst_off;
                const char *src = src0 + ks * (BK * 2);
#pragma unroll
                for (int i = 0; i < NR; i++)
                    if (off[i] >= 0) cp_async16(sb + i * (RSTEP * 128), src + off[i], pol_t);
                cp_async_commit();
                p.advance(STAGES);
            }
            if (!ok) break;
            // the next item's row indices travel while the last stages of this one land
            len = next_item(off_next);
            static_assert(LAG == 2 || LAG == 3, "copy lag");
            if (LAG == 3) hand_over(std::integral_constant<int, 2>{});
            hand_over(std::integral_constant<int, 1>{});
            hand_over(std::integral_constant<int, 0>{});
#pragma unroll
            for (int i = 0; i < NR; i++) off[i] = off_next[i];
        }
        cp_async_wait<0>();
    } else if (warp == 3 && !gathering) {
        // ---------------------------------------------------------- token producer, TMA
        PipeState p, wr;
        const uint64_t pol_t = l2_policy_evict_last();
        int ready_group = -1;
        bool ok = true;
        while (ok) {
            ok = xwait_warp<PAIR>(ifull_bar(wr.stage), wr.phase, ab);
            if (!ok) break;
            const int row0 = uniform_i32(ring[wr.stage].row0), len = uniform_i32(ring[wr.stage].len), expert = uniform_i32(ring[wr.stage].expert);
            if (elect_one()) arrive_lead(iempty_bar(wr.stage));
            wr.advance(X_RING);
            if (len < 0) break;
            if (a.ready && expert / a.group_size != ready_group) {
                // expert parallelism: this expert's rows are being written by other GPUs while the
                // kernel runs; wait (bounded, polling gently) until its whole group has arrived
                const int grp = expert / a.group_size;
                const uint32_t want = a.need_blocks ? (uint32_t)a.need_blocks : (uint32_t)a.need[grp];
                const uint64_t t0 = globaltimer_ns();
                while (!__all_sync(0xffffffffu, ld_acquire_sys_u32(a.ready + grp) == want)) {
                    __nanosleep(500);
                    if (__any_sync(0xffffffffu, *abort_flag || globaltimer_ns() - t0 > WAIT_LIMIT_NS)) {
                        if (elect_one()) ab.raise(OMNI_ST_TIMEOUT | OMNI_ST_TIMEOUT_ARRIVAL);
                        ok = false;
                        break;
                    }
                }
                if (!ok) break;
                fence_proxy_async_all();          // the rows are read next by TMA (async proxy)
                ready_group = grp;
            }
            const int share = ((len + 15) & ~15) / CTAS;
            const int bi = tok_box_index(share);
            const uint32_t bytes = tok_box_bytes(bi);
            for (int ks = 0; ks < KSTAGES; ks++) {
                ok = xwait_warp<false>(empty_bar(p.stage), p.phase ^ 1u, ab);
                if (!ok) break;
                if (elect_one()) {
                    if (leader) {
                        armed_t[p.stage] = (int)p.phase;
                        mbar_expect_tx(full_bar(p.stage), CTAS * bytes);
                    }
                    xtma_2d<CTAS>(tok_base + p.stage * C::T_BYTES, &tm_tok.m[bi], ks * BK, row0 + (int)rank * share,
                                  lead(full_bar(p.stage)), pol_t);
                }
                p.advance(STAGES);
            }
        }
    } else if (warp == 1 && leader) {
        // ---------------------------------------------------------- MMA issuer (first CTA of the pair)
        PipeState p, wr;
        bool ok = true;
        for (int it = 0; ok; it++) {
            ok = xwait_warp<PAIR>(ifull_bar(wr.stage), wr.phase, ab);
            if (!ok) break;
            const int len = uniform_i32(ring[wr.stage].len);
            if (elect_one()) mbar_arrive(iempty_bar(wr.stage));
            wr.advance(X_RING);
            if (len < 0) break;
            const int n_mma = (len + 15) & ~15;
            const uint32_t idesc = idesc_bf16(128 * CTAS, n_mma);
            const int buf = it & 1;
            ok = xwait_warp<false>(aempty_bar(buf), ((uint32_t)(it >> 1) & 1u) ^ 1u, ab);
            if (!ok) break;
            tc_fence_after();
            const uint32_t d0 = tmem_base + buf * 256;
            for (int ks = 0; ks < KSTAGES; ks++) {
                ok = xwait_warp<false>(full_bar(p.stage), p.phase, ab);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t da = smem_desc_sw128(smem_base + p.stage * C::W_BYTES);
                    const uint64_t db = smem_desc_sw128(tok_base + p.stage * C::T_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / 16; k++) xmma<CTAS>(d0, da + 2u * k, db + 2u * k, idesc, (ks | k) ? 1u : 0u);
                    xcommit<CTAS>(empty_bar(p.stage));     // what was staged is free (in both CTAs) once these MMAs have read it
                    if (ks == KSTAGES - 1) xcommit<CTAS>(afull_bar(buf));        // accumulator complete, in both CTAs
                }
                __syncwarp();
                p.advance(STAGES);
            }
        }
        // Whatever happened, wait (bounded) until every MMA issued by this warp's elected thread has
        // retired before tensor memory is released.
        if (elect_one()) {
            xcommit<CTAS>(drain_bar);
            const uint64_t t0 = globaltimer_ns();
            while (!mbar_try_wait(drain_bar, 0) && globaltimer_ns() - t0 < WAIT_LIMIT_NS) {}
        }
        __syncwarp();
    } else if (COPY && warp >= 16) {
        // ---------------------------------------------------------- dispatch of this rank's token rows
        // (expert parallelism): each token once per owner rank, plain peer stores into the owners'
        // receive buffers, group by group, each group announced on the owner's arrival counter --
        // which the token producers above, here and on the other ranks, wait for.  Virtual block =
        // the copy warps of one CTA.
        const int nvb = (int)gridDim.x - (int)gridDim.x % a.pe.world;
        if ((int)blockIdx.x < nvb)
            ep_dispatch_dedup(a.pe, a.send, (int)blockIdx.x, nvb, warp - 16, X_COPY_THREADS / 32, lane, threadIdx.x == X_THREADS + X_GATHER_THREADS,
                              [] { named_bar_sync(3, X_COPY_THREADS); });
    } else if (warp >= 4 && warp < 12) {
        // ---------------------------------------------------------- epilogue: TMEM -> registers -> shared -> HBM
        // The two halves split an item's 32-row chunks and do not wait for one another.  A half's four
        // warps (one per TMEM quadrant, i.e. 32 accumulator rows each) write a chunk's columns into
        // a shared-memory tile, meet at a named barrier and store whole row pieces; the next chunk
        // uses the other of two tiles, so one barrier per chunk is enough.  They also meet before
        // the first chunk of an item: a warp whose wait ran out says so there and all four leave
        // together.
        const int q = warp & 3;                       // TMEM lane quadrant this warp may read
        const int half = (warp - 4) >> 2;
        const int th = ((warp - 4) & 3) * 32 + lane;  // thread index inside the half (0..127)
        // The combine reads d next: what of it is still in L2 then need not come back from memory.  us per block without and
        // with, both in turn under the power limit: 1030 and 2048 tokens the same, 4096 437.9 -> 436.4, 12000 1048.7 -> 1039.8, 16384
        // 1380 -> 1370.
        const uint64_t pol_d = l2_policy_evict_last();
        PipeState wr;
        for (int it = 0;; it++) {
            int row0 = 0, len = 0, m = 0;
            bool got = xwait_warp<PAIR>(ifull_bar(wr.stage), wr.phase, ab);
            if (got) {
                row0 = ring[wr.stage].row0; len = ring[wr.stage].len; m = ring[wr.stage].m;
                __syncwarp();
                if (lane == 0) arrive_lead(iempty_bar(wr.stage));
                wr.advance(X_RING);
            }
            const bool stop = got && len < 0;
            const int buf = it & 1;
            const int nchunk = (len + 31) >> 5;
            const int c_lo = half ? (nchunk + 1) >> 1 : 0, c_hi = half ? nchunk : (nchunk + 1) >> 1;
            if (got && !stop) got = xwait_warp<false>(afull_bar(buf), (uint32_t)(it >> 1) & 1u, ab);
            if (!warps_meet(epi_quit + 2 * half, it, got, [&] { named_bar_sync(1 + half, 128); }) || stop) break;
            tc_fence_after();
            const uint32_t t0 = tmem_base + ((uint32_t)(q * 32) << 16) + buf * 256;
            const int m_cta = m * CTAS + (int)rank;
            if (c_lo == c_hi) {                       // nothing for this half: hand tensor memory back
                tc_fence_before();
                __syncwarp();
                if (lane == 0) arrive_lead(aempty_bar(buf));
            }
            for (int c = c_lo; c < c_hi; c++) {
                auto release = [&] {
                    // tensor memory goes back to the MMA thread before the last stores to HBM start
                    if (c != c_hi - 1) return;
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) arrive_lead(aempty_bar(buf));
                };
                if constexpr (MODE == X_OPROJ) {
                    uint32_t v[32];
                    tmem_ld32(t0 + c * 32, v);
                    // added into the FP32 residual: a warp's 32 lanes are 32 consecutive columns of one row;
                    // all loads of the chunk before its stores, so that they are in flight together
                    float *xr = a.resid + (long)(row0 + c * 32) * M::OUT_COLS + m_cta * M::OUTC + q * 32 + lane;
                    float old[32];
#pragma unroll
                    for (int j = 0; j < 32; j++) old[j] = c * 32 + j < len ? xr[(long)j * M::OUT_COLS] : 0.f;
                    tmem_ld_wait();
                    release();
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (c * 32 + j < len) xr[(long)j * M::OUT_COLS] = old[j] + __uint_as_float(v[j]);
                } else {
                    // Row j of the tile is token c*32 + j; its 16-byte pieces sit at piece ^ (j & 7), so that neither
                    // the stmatrix rows (eight tokens, same piece) nor the reads below meet in a bank.
                    constexpr int PITCH = M::OUTC * 2, PIECES = M::OUTC / 8;
                    uint8_t *const tile = out_tile + (half * 2 + ((c - c_lo) & 1)) * C::CHUNK_BYTES;
                    uint32_t lo[16], hi[16];
                    tmem_ld_16x32(t0 + c * 32, lo);
                    tmem_ld_16x32(t0 + c * 32 + (16u << 16), hi);
                    tmem_ld_wait();
                    release();
                    const int tok = ((lane >> 4) << 3) | (lane & 7), sub8 = (lane >> 3) & 1;
                    const uint32_t row_addr = smem_u32(tile) + tok * PITCH;
                    auto store16 = [&](const uint32_t (&p)[8], int piece) {     // 16 output columns of all 32 tokens
                        const uint32_t at = row_addr + (((piece + sub8) ^ (tok & 7)) << 4);
                        stmatrix_x4_trans(at, p[0], p[1], p[2], p[3]);
                        stmatrix_x4_trans(at + 16 * PITCH, p[4], p[5], p[6], p[7]);
                    };
                    if constexpr (MODE == X_GATEUP) {
                        uint32_t p[8];                    // lanes 0..15 of the quadrant are gate rows, 16..31 the up rows of the same columns
#pragma unroll
                        for (int i = 0; i < 8; i++)
                            p[i] = pack_bf16(silu_mul(__uint_as_float(lo[2 * i]), __uint_as_float(hi[2 * i])),
                                             silu_mul(__uint_as_float(lo[2 * i + 1]), __uint_as_float(hi[2 * i + 1])));
                        store16(p, q * 2);
                    } else {
                        uint32_t p[8];
#pragma unroll
                        for (int i = 0; i < 8; i++) p[i] = pack_bf16(__uint_as_float(lo[2 * i]), __uint_as_float(lo[2 * i + 1]));
                        store16(p, q * 4);
#pragma unroll
                        for (int i = 0; i < 8; i++) p[i] = pack_bf16(__uint_as_float(hi[2 * i]), __uint_as_float(hi[2 * i + 1]));
                        store16(p, q * 4 + 2);
                    }
                    named_bar_sync(1 + half, 128);        // the four quadrants have written their columns
                    constexpr int LANES_PER_ROW = PIECES;                        // 8 (gate/up) or 16
                    const int sub = th % LANES_PER_ROW;
#pragma unroll
                    for (int i = 0; i < 32 * LANES_PER_ROW / 128; i++) {
                        const int rr = th / LANES_PER_ROW + i * (128 / LANES_PER_ROW), r = c * 32 + rr;
                        if (r >= len) break;
                        const uint4 val = *reinterpret_cast<const uint4 *>(tile + rr * PITCH + ((sub ^ (rr & 7)) << 4));
                        __nv_bfloat16 *dst_row;
                        if (MODE == X_DOWN && a.rowinfo) {
                            const int info = __ldg(a.rowinfo + row0 + r);
                            dst_row = reinterpret_cast<__nv_bfloat16 *>(a.pe.dret[info >> 20]) + (long)(info & 0xfffff) * M::OUT_COLS;
                        } else {
                            dst_row = a.out + (long)(row0 + r) * M::OUT_COLS;
                        }
                        if (MODE == X_DOWN && !a.rowinfo) st_global_hint(dst_row + m_cta * M::OUTC + sub * 8, val, pol_d);
                        else *reinterpret_cast<uint4 *>(dst_row + m_cta * M::OUTC + sub * 8) = val;
                    }
                }
            }
        }
    }

    // ---------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0) {
        // a wait ran out; of a pair the first CTA knows what both announced
        copies_land(armed_w, 2 * STAGES, [&](int i, int parity) { return mbar_try_wait(full_bar(i % STAGES), (uint32_t)parity) != 0; },
                    globaltimer_ns, LAND_LIMIT_NS, LAND_SETTLE_NS);
    }
    // neither CTA of a pair may leave while the other's MMAs can still read its shared memory
    if (PAIR) cluster_sync_all(); else __syncthreads();
    if (warp == 2) { tc_fence_after(); xtmem_dealloc<CTAS>(tmem_base, 512); }
}

}  // namespace

// ====================================================================== launchers
namespace {

template <int MODE, int CTAS, bool COPY>
cudaError_t launch_pair(const CUtensorMap *tm_w, const CUtensorMap *tm_tok, const XArgs &args, int n_sm, cudaStream_t s) {
    TokMaps tok;
    for (int i = 0; i < OMNI_TOK_BOXES; i++) tok.m[i] = tm_tok[i];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n_sm - n_sm % CTAS));
    cfg.blockDim = dim3(x_threads<MODE, COPY>());
    cfg.dynamicSmemBytes = XCfg<MODE, CTAS>::TOTAL_BYTES;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (CTAS == 2) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 2; attr[n].val.clusterDim.y = 1; attr[n].val.clusterDim.z = 1;
        n++;
    }
    if (omni_dependent_launch_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        n++;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, expert_pair_kernel<MODE, CTAS, COPY>, *tm_w, tok, args);
}

template <int MODE, int CTAS, bool COPY>
cudaError_t set_smem() {
    return cudaFuncSetAttribute(expert_pair_kernel<MODE, CTAS, COPY>, cudaFuncAttributeMaxDynamicSharedMemorySize, XCfg<MODE, CTAS>::TOTAL_BYTES);
}

}  // namespace

extern "C" {

cudaError_t omni_expert_configure(void) {
    cudaError_t e;
    if ((e = set_smem<X_GATEUP, 1, false>()) != cudaSuccess) return e;
    if ((e = set_smem<X_GATEUP, 2, false>()) != cudaSuccess) return e;
    if ((e = set_smem<X_GATEUP, 1, true>()) != cudaSuccess) return e;
    if ((e = set_smem<X_GATEUP, 2, true>()) != cudaSuccess) return e;
    if ((e = set_smem<X_DOWN, 1, false>()) != cudaSuccess) return e;
    if ((e = set_smem<X_QKV, 2, false>()) != cudaSuccess) return e;
    if ((e = set_smem<X_OPROJ, 2, false>()) != cudaSuccess) return e;
    return set_smem<X_DOWN, 2, false>();
}

cudaError_t omni_launch_gateup_pair(int ctas, const CUtensorMap *tm_w4, const CUtensorMap *tm_x, const omni_sort_state st,
                                    void *h, const uint32_t *ready, const int32_t *need, int group_size,
                                    const void *gather_src, const int32_t *gather_rows, const omni_ep_peers *dispatch_to,
                                    const omni_ep_send *send, int early_dependents, int n_sm, cudaStream_t s) {
    XArgs a = {};
    a.ttiles = st.ttiles; a.n_ttiles = st.n_ttiles; a.work_counter = st.sched; a.out = (__nv_bfloat16 *)h; a.status = st.status;
    a.ready = ready; a.need = need; a.group_size = group_size > 0 ? group_size : 1;
    a.gather_src = (const __nv_bfloat16 *)gather_src; a.gather_rows = gather_rows;
    a.early_dependents = early_dependents;
    if (dispatch_to) {
        const int grid = n_sm - n_sm % ctas;
        a.pe = *dispatch_to;
        a.send = *send;
        a.need_blocks = grid - grid % dispatch_to->world;       // every rank launches the same grid
        return ctas == 2 ? launch_pair<X_GATEUP, 2, true>(tm_w4, tm_x, a, n_sm, s) : launch_pair<X_GATEUP, 1, true>(tm_w4, tm_x, a, n_sm, s);
    }
    return ctas == 2 ? launch_pair<X_GATEUP, 2, false>(tm_w4, tm_x, a, n_sm, s) : launch_pair<X_GATEUP, 1, false>(tm_w4, tm_x, a, n_sm, s);
}

cudaError_t omni_launch_down_pair(int ctas, const CUtensorMap *tm_w, const CUtensorMap *tm_h, const omni_sort_state st,
                                  void *d, const omni_ep_peers *return_to, const int32_t *rowinfo, int early_dependents,
                                  const void *weights, int n_sm, cudaStream_t s) {
    XArgs a = {};
    a.weights = (const char *)weights;
    a.ttiles = st.ttiles; a.n_ttiles = st.n_ttiles; a.work_counter = st.sched + 1;
    a.out = (__nv_bfloat16 *)d; a.status = st.status; a.group_size = 1;
    if (return_to) { a.pe = *return_to; a.rowinfo = rowinfo; }
    a.early_dependents = early_dependents;
    return ctas == 2 ? launch_pair<X_DOWN, 2, false>(tm_w, tm_h, a, n_sm, s) : launch_pair<X_DOWN, 1, false>(tm_w, tm_h, a, n_sm, s);
}

// The dense projections of the attention half on the same kernel: tm_w is the weight matrix
// [OUT_COLS][K] with a 64 x 128 box, tm_tok the token operand.  The T token rows are cut into near-equal tiles.
cudaError_t omni_launch_dense_pair(int which, const CUtensorMap *tm_w, const CUtensorMap *tm_tok, int T, void *out_bf16, float *resid,
                                   uint32_t *status, int early_dependents, int n_sm, cudaStream_t s) {
    XArgs a = {};
    a.out = (__nv_bfloat16 *)out_bf16; a.resid = resid; a.status = status; a.group_size = 1;
    a.early_dependents = early_dependents;
    a.dense_rows = T;
    // Tiles: the fewest rounds of the pairs of SMs weighted by what an item of that many rows costs: about n/2 clocks per K step
    // of 16, and the weight rows, which come through the SM once per item however few tokens they meet.  (With a floor of
    // 96 rows in place of that the q|k|v projection of 1030 tokens took three rounds of 96 rows where two of 160
    // do: attention half 74.0 -> 69.0 us, both in turn; 300, 2048 and 4096 tokens the same within 1 %.)
    const int blocks = (which == 0 ? OMNI_QKV : OMNI_H) / 256, pairs = n_sm / 2;
    long best = -1;
    for (int nt = (T + OMNI_TILE_N - 1) / OMNI_TILE_N; nt <= T; nt++) {
        const int rows = ((T + nt - 1) / nt + 15) & ~15;
        const long rounds = ((long)nt * blocks + pairs - 1) / pairs, cost = rounds * (rows + DENSE_ITEM);
        if (best < 0 || cost < best) { best = cost; a.dense_tiles = nt; }
        if (rows <= DENSE_MIN) break;
    }
    return which == 0 ? launch_pair<X_QKV, 2, false>(tm_w, tm_tok, a, n_sm, s) : launch_pair<X_OPROJ, 2, false>(tm_w, tm_tok, a, n_sm, s);
}

}  // extern "C"
