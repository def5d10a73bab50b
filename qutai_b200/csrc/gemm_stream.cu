// Expert products for few rows per expert (decoding, short prompts), where the pass over the weights is the work:
// C[rows, N] = A[rows, K] . B_e formed as its transpose, so that the WEIGHT tile is the 128-row operand of the MMA and an
// expert's rows are its columns (N = 16 .. 128, as many as there are).
//
// The kernel for many rows (gemm_tcgen05.cu) gives every expert tiles of 256 rows: an expert with six rows still costs
// the tensor time of 256 and stages 128 rows of activations beside every 128 rows of weights.  Here both follow the
// expert's own row count, and what bounds a product is HBM: 96 KiB of weight tiles in flight per SM (STREAM_NT), 128 KiB in
// the other two, more for few tokens (few_tokens).  64 rows over 64 experts, top 6, 2048 x 1408: SwiGLU 144 -> 113 us (738 MB: 6.5 TB/s), down product 72 -> 60.
//
// One persistent CTA per SM, or per tile where those are fewer, 6 warps: warp 0 asks TMA for the tiles, warp 1 issues the MMAs, warps 2-5 convert the
// accumulators (lane = output column, TMEM column = row of the expert) and store them; two accumulator sets, so a
// tile's epilogue runs beside the next tile's main loop.
//   STREAM_SWIGLU   G, U, H from X: a stage holds 64 columns of a gate tile and of the up tile beside it
//   STREAM_NT       C = A . B_e^T, B stacked [E * N, K]
//   STREAM_NT2      the same with 256 output columns per tile, so that a stage of activations serves two weight tiles: for
//                   experts of many rows, whose activations are as many bytes as a weight tile
// Every wait is bounded (status codes 111 .. 113).
#include "common.cuh"
#include "tc_ptx.cuh"

namespace qmoe {
namespace {

constexpr int SM_ROWS = 128, SK = 64;                  // weight rows of a tile, contraction columns of a stage
constexpr int W_BYTES = SM_ROWS * SK * 2;              // 16 KiB
constexpr int X_BOX = 32, X_BOX_BYTES = X_BOX * SK * 2;  // activations arrive in boxes of 32 rows
constexpr int X_BYTES = kRowPad * SK * 2;              // at most 128 rows: 16 KiB
constexpr int STREAM_THREADS = 192;
constexpr uint32_t STREAM_TMEM = 512;                  // two sets of two 128-column accumulators

enum { STREAM_SWIGLU = 0, STREAM_NT = 1, STREAM_NT2 = 2 };
enum { STATUS_STREAM_PRODUCER = 111, STATUS_STREAM_MMA = 112, STATUS_STREAM_EPILOGUE = 113 };

// FEW: at most X_BOX rows per expert, one box of activations per stage, and the room for more stages
template <int MODE, bool FEW> struct StreamCfg {
    static constexpr int W_TILES = MODE == STREAM_NT ? 1 : 2;
    static constexpr int MOST_ROWS = FEW ? X_BOX : kRowPad;                       // of an expert in a tile; more rows are more tiles
    static constexpr int STAGE_BYTES = W_TILES * W_BYTES + (FEW ? X_BOX_BYTES : X_BYTES);
    static constexpr int STAGES = MODE == STREAM_NT ? (FEW ? 11 : 6) : FEW ? 6 : 4;
    static constexpr int COLUMNS = MODE == STREAM_NT2 ? 2 * SM_ROWS : SM_ROWS;    // output columns of a tile
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
};

struct alignas(64) StreamParams {
    CUtensorMap map_w, map_w2;     // weights (gate and up, or the only one)
    CUtensorMap map_x;             // activations in the dispatched layout
    const int* offsets;
    const int* counts;
    int* status;
    __nv_bfloat16* out0;           // SWIGLU: G; NT: C
    __nv_bfloat16* out1;           // SWIGLU: U
    __nv_bfloat16* out2;           // SWIGLU: H
    int experts, m_tiles, N, K;
    int early;                     // what lies two launches back wrote the tables and the weights: see the wait
    int let_next;                  // the next kernel is the down product of the same call: it may start early
    int pad_rows;                  // zero every pad row; else those from `columns` on are left as they are
};

// `columns`: rows of the expert in this tile, rounded up to 16; `end`: with the pad rows that are this tile's to fill
struct StreamTile { int expert, n0, row0, columns, end; };

// tiles of expert e: m_tiles weight tiles x its chunks of most_rows rows, the chunks of one weight tile side by side (the second
// finds the weights in L2)
// (first, row0, rows: each expert's first tile, first dispatched row and rows, in shared memory; most_rows: what a stage has room for)
__device__ __forceinline__ StreamTile stream_tile(const StreamParams& p, const int* first, const int* row0, const int* rows, int t, int columns, int most_rows) {
    int lo = 0, hi = p.experts;        // largest e with first[e] <= t
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (first[mid] <= t) lo = mid; else hi = mid;
    }
    const int chunks = (first[lo + 1] - first[lo]) / p.m_tiles, local = t - first[lo], chunk = local % chunks;
    StreamTile tile;
    tile.expert = lo;
    tile.n0 = local / chunks * columns;
    tile.row0 = row0[lo] + chunk * most_rows;
    const int left = rows[lo] - chunk * most_rows;
    tile.columns = left >= most_rows ? most_rows : (left + kStreamPad - 1) / kStreamPad * kStreamPad;
    tile.end = left > most_rows ? most_rows : kRowPad - chunk * most_rows % kRowPad;      // the last chunk fills up to the next 128
    return tile;
}

__device__ __forceinline__ float logistic(float v) {   // 1 / (1 + 2^(-v log2 e)) as in the kernel for many rows
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-1.4426950408889634f * v));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return r;
}

template <int MODE, bool FEW>
__global__ void __launch_bounds__(STREAM_THREADS, 1)
stream_gemm_kernel(const __grid_constant__ StreamParams p) {
    using Config = StreamCfg<MODE, FEW>;
    constexpr int STAGES = Config::STAGES, STAGE_BYTES = Config::STAGE_BYTES, W_TILES = Config::W_TILES;
    extern __shared__ uint8_t smem_raw[];
    __shared__ int s_first[kMaxExperts + 1], s_row0[kMaxExperts], s_rows[kMaxExperts];     // see stream_tile
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, bars = base + STAGES * STAGE_BYTES;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
    auto tfull_bar = [&](int a) { return bars + 8u * (2 * STAGES + a); };
    auto tempty_bar = [&](int a) { return bars + 8u * (2 * STAGES + 2 + a); };

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(tfull_bar(a), 1); mbar_init(tempty_bar(a), 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        prefetch_map(&p.map_w); prefetch_map(&p.map_w2); prefetch_map(&p.map_x);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(STREAM_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // `early`: the kernel before is this call's own (the permutation, or the product that forms H), writes neither tables nor weights and lets
    // this one start behind its own wait, so whatever wrote those lies at least two launches back and is complete.  The tables and the first
    // stages' weights are then fetched beside the kernel before; what that one writes (the activations), and whatever this one writes, waits.
    // us a replay with neither product early, the up product, and both, on one stream, then of two at a time, then of four: 4 rows, 8 experts,
    // 1024 x 2816, 38.4 35.8 33.0, 45.7 45.3 46.1, 70.1 67.5 67.5; 16 rows, 4 experts, 512 x 264, 24.7 24.7 20.6, 24.7 24.7 22.6, 27.9 26.6 24.4; 1 row,
    // 32 experts, 2048 x 1408, 45.0 41.9 41.1, 55.3 54.2 59.2, 86.4 84.2 84.3.  CTAs that wait for the tail of the up product keep other streams'
    // kernels from their SMs, which two streams of short tails feel most; 64 rows over 64 experts, on several streams 158.6 without the down product and
    // 160.6 with it.  So the down product starts early for few tokens alone.
    if (!p.early) chain_wait();
    // The tables in one round trip to L2: a thread per expert loads, a warp sums up (every thread adding up the counts before its
    // expert is a chain of L2 latencies: 64 rows over 64 experts, replayed, L2 flushed before every call, 217 us and 215 like this).
    for (int e = threadIdx.x; e < p.experts; e += STREAM_THREADS) {
        const int count = load_l2(p.counts + e);
        s_rows[e] = count;
        s_row0[e] = load_l2(p.offsets + e);
        s_first[e + 1] = (count + Config::MOST_ROWS - 1) / Config::MOST_ROWS * p.m_tiles;
    }
    __syncthreads();
    if (warp == 0) {
        int before = 0;
        for (int e0 = 0; e0 < p.experts; e0 += 32) {
            int sum = e0 + lane < p.experts ? s_first[e0 + lane + 1] : 0;
#pragma unroll
            for (int step = 1; step < 32; step *= 2) {
                const int other = __shfl_up_sync(0xffffffffu, sum, step);
                if (lane >= step) sum += other;
            }
            if (e0 + lane < p.experts) s_first[e0 + lane + 1] = before + sum;
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) s_first[0] = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem_base;
    const int total = s_first[p.experts], kblocks = (p.K + SK - 1) / SK;
    volatile int* abort_flag = &s_abort;
    auto gave_up = [&](int code) { if (!*abort_flag) { *abort_flag = 1; atomicExch(p.status, code); } };

    if (warp == 0) {
        auto ask_weights = [&](int stage, int kb, int w_row) {
            const uint32_t w = base + stage * STAGE_BYTES, bar = full_bar(stage);
            tma_load_2d(&p.map_w, w, bar, kb * SK, w_row);
            if (MODE == STREAM_SWIGLU) tma_load_2d(&p.map_w2, w + W_BYTES, bar, kb * SK, w_row);
            if (MODE == STREAM_NT2) tma_load_2d(&p.map_w, w + W_BYTES, bar, kb * SK, w_row + SM_ROWS);
        };
        auto ask_rows = [&](int stage, int kb, int row0, int boxes) {
            const uint32_t x = base + stage * STAGE_BYTES + W_TILES * W_BYTES, bar = full_bar(stage);
            for (int j = 0; j < boxes; ++j) tma_load_2d(&p.map_x, x + j * X_BOX_BYTES, bar, kb * SK, row0 + j * X_BOX);
        };
        int ahead = 0;       // k-blocks of the first tile whose weights were asked for before the wait
        StreamTile first_tile = {};
        if (p.early) {
            if ((int)blockIdx.x < total) {
                first_tile = stream_tile(p, s_first, s_row0, s_rows, (int)blockIdx.x, Config::COLUMNS, Config::MOST_ROWS);
                ahead = kblocks < STAGES ? kblocks : STAGES;
            }
            const int boxes = (first_tile.columns + X_BOX - 1) / X_BOX;
            if (lane == 0)
                for (int kb = 0; kb < ahead; ++kb) {      // the stages are empty
                    mbar_expect_tx(full_bar(kb), W_TILES * W_BYTES + boxes * X_BOX_BYTES);
                    ask_weights(kb, kb, first_tile.expert * p.N + first_tile.n0);
                }
            chain_wait();
            if (lane == 0)
                for (int kb = 0; kb < ahead; ++kb) ask_rows(kb, kb, first_tile.row0, boxes);
        }
        if (lane == 0) {
            int stage = ahead == STAGES ? 0 : ahead;
            uint32_t phase = ahead == STAGES ? 1 : 0;
            for (int t = blockIdx.x; t < total && !*abort_flag; t += gridDim.x, ahead = 0) {
                const StreamTile tile = stream_tile(p, s_first, s_row0, s_rows, t, Config::COLUMNS, Config::MOST_ROWS);
                const int boxes = (tile.columns + X_BOX - 1) / X_BOX;
                for (int kb = ahead; kb < kblocks; ++kb) {
                    if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag)) { gave_up(STATUS_STREAM_PRODUCER); break; }
                    mbar_expect_tx(full_bar(stage), W_TILES * W_BYTES + boxes * X_BOX_BYTES);
                    ask_weights(stage, kb, tile.expert * p.N + tile.n0);
                    ask_rows(stage, kb, tile.row0, boxes);
                    if (++stage == STAGES) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        if (p.early) chain_wait();
        if (p.let_next) chain_next();      // the tensor memory is this block's
        // One elected lane walks the blocks and looks at the next stage's barrier before the last MMA of this one, while the tensor pipe has work
        // queued: an MMA of 128 weight rows takes 66 cycles for up to 32 columns and 81 for 128, eight of them 530 .. 650 per k-block, and the
        // waits, votes and elections of a whole warp came on top (4 rows, 8 experts, 1024 x 2816: 42.9 us a call, like this 40.6).
        if (elect_one()) {
            int stage = 0, iter = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int t = blockIdx.x; ok && t < total; t += gridDim.x, ++iter) {
                const StreamTile tile = stream_tile(p, s_first, s_row0, s_rows, t, Config::COLUMNS, Config::MOST_ROWS);
                const uint32_t idesc = make_idesc<false, false, SM_ROWS>(tile.columns), acc = tmem + (uint32_t)(iter & 1) * 256;
                ok = mbar_wait(tempty_bar(iter & 1), ((uint32_t)(iter >> 1) & 1u) ^ 1u, abort_flag);
                tc_fence_after();
                bool ready = false;      // the stage of this k-block was seen full while the one before it was issued
                for (int kb = 0; ok && kb < kblocks; ++kb) {
                    if (!ready) ok = mbar_wait(full_bar(stage), phase, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t w = base + stage * STAGE_BYTES, x = w + W_TILES * W_BYTES;
                    int next_stage = stage + 1;
                    uint32_t next_phase = phase;
                    if (next_stage == STAGES) { next_stage = 0; next_phase ^= 1u; }
#pragma unroll
                    for (int which = 0; which < W_TILES; ++which)
#pragma unroll
                        for (int kk = 0; kk < SK / 16; ++kk) {
                            if (which == W_TILES - 1 && kk == SK / 16 - 1) ready = kb + 1 < kblocks && mbar_try(full_bar(next_stage), next_phase);
                            umma_bf16(acc + which * 128, make_desc(w + which * W_BYTES + kk * 32, 16, 1024), make_desc(x + kk * 32, 16, 1024), idesc,
                                      (kb | kk) ? 1u : 0u);
                        }
                    umma_commit(empty_bar(stage));
                    if (kb == kblocks - 1) umma_commit(tfull_bar(iter & 1));
                    stage = next_stage; phase = next_phase;
                }
            }
            if (!ok) gave_up(STATUS_STREAM_MMA);
        }
    } else {
        if (p.early) chain_wait();
        const int quad = warp & 3;
        int iter = 0;
        for (int t = blockIdx.x; t < total; t += gridDim.x, ++iter) {
            const StreamTile tile = stream_tile(p, s_first, s_row0, s_rows, t, Config::COLUMNS, Config::MOST_ROWS);
            const int a = iter & 1, n = tile.n0 + quad * 32 + lane;
            if (!__all_sync(0xffffffffu, mbar_wait(tfull_bar(a), (uint32_t)(iter >> 1) & 1u, abort_flag))) {
                if (lane == 0) gave_up(STATUS_STREAM_EPILOGUE);
                break;
            }
            tc_fence_after();
            const uint32_t acc = tmem + (uint32_t)a * 256 + ((uint32_t)(quad * 32) << 16);
            const long long at = (long long)tile.row0 * p.N + n;
#pragma unroll 1
            for (int c = 0; c < tile.columns; c += 16) {      // a store instruction covers 32 consecutive columns of one row
                uint32_t v0[16], v1[16];
                tmem_ld16(acc + c, v0);
                if (W_TILES == 2) tmem_ld16(acc + 128 + c, v1);
                tmem_ld_wait();
                if (n < p.N) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        const long long to = at + (long long)(c + e) * p.N;
                        if (MODE == STREAM_SWIGLU) {
                            // H from the rounded G and U, which are what the backward reads
                            const __nv_bfloat16 gb = __float2bfloat16_rn(__uint_as_float(v0[e])), ub = __float2bfloat16_rn(__uint_as_float(v1[e]));
                            const float g = __bfloat162float(gb);
                            p.out0[to] = gb;
                            p.out1[to] = ub;
                            p.out2[to] = __float2bfloat16_rn(g * logistic(g) * __bfloat162float(ub));
                        } else {
                            p.out0[to] = __float2bfloat16_rn(__uint_as_float(v0[e]));
                            if (MODE == STREAM_NT2 && n + SM_ROWS < p.N) p.out0[to + SM_ROWS] = __float2bfloat16_rn(__uint_as_float(v1[e]));
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty_bar(a));
            if (p.pad_rows && n < p.N) {
                const __nv_bfloat16 zero = __float2bfloat16_rn(0.f);
                for (int c = tile.columns; c < tile.end; ++c) {
                    const long long to = at + (long long)c * p.N;
                    p.out0[to] = zero;
                    if (MODE == STREAM_SWIGLU) { p.out1[to] = zero; p.out2[to] = zero; }
                    if (MODE == STREAM_NT2 && n + SM_ROWS < p.N) p.out0[to + SM_ROWS] = zero;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (s_abort) {   // copies and MMAs in flight get a bounded time to land before shared memory and TMEM go away
        const unsigned long long start = global_ns();
        while (global_ns() - start < 2000000ull) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(STREAM_TMEM) : "memory");
    }
}

template <int MODE, bool FEW = false>
int stream_launch(const StreamParams& p, const qmoe_route_t* r, cudaStream_t stream) {
    static bool configured[64] = {};      // per device, like the kernels of gemm_tcgen05.cu
    constexpr int SMEM_BYTES = StreamCfg<MODE, FEW>::SMEM_BYTES;
    static_assert(SMEM_BYTES + 3 * 4 * (kMaxExperts + 1) + 16 <= 227 * 1024, "the stages and the tables exceed the shared memory of a block");
    int dev = 0;
    QMOE_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail_arg("device ordinal beyond 63");
    if (!configured[dev]) {
        QMOE_CUDA(cudaFuncSetAttribute(stream_gemm_kernel<MODE, FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        configured[dev] = true;
    }
    // No more CTAs than there can be tiles (a caller's own tables may hold more: a CTA walks them in steps of the grid).  One that finds none would
    // hold its SM until the kernel before is done: 16 rows, 4 experts, 512 x 264, replayed on four streams 30.6 us with a CTA for every SM and
    // 24.4 like this, 1 row, 32 experts, 2048 x 1408, 90.1 and 84.3, on one stream even.
    const long long rows = r->tokens * r->top_k, most = ((rows < p.experts ? rows : p.experts) + rows / StreamCfg<MODE, FEW>::MOST_ROWS) * p.m_tiles;
    chained(stream_gemm_kernel<MODE, FEW>, most < sm_count() ? (int)most : sm_count(), STREAM_THREADS, SMEM_BYTES, stream, p);
    count_tensor_core_launch();
    QMOE_LAUNCH_CHECK("stream_gemm_kernel");
    return 0;
}

// The form with more stages: up to X_BOX tokens (a routing sends a token to an expert once, so that no expert has more rows; tables that a caller
// filled may, which takes tiles of X_BOX rows each), and with the experts that uniform load reaches on average at most two tiles per SM.  There a tile's time is what one SM has on its way; with more tiles
// HBM is the limit, and the more is asked for at once the less it gives.  us a call, 128 KiB of weights in flight per SM and 192: 8 experts,
// 1024 x 2816, 4 rows 40.9 and 40.6, 32 rows 52.2 and 51.4, 1 row of 4096 x 2816 67.9 and 62.8, 64 experts, 2048 x 1408, 1 row 46.9 and 45.1, but
// 16 rows 169.9 and 172.8, 32 rows 196.6 and 203.2.
bool few_tokens(const qmoe_route_t* r, int experts, long long tiles_per_expert) {
    if (r->tokens > X_BOX) return false;
    const double hit = r->top_k < experts ? (double)r->top_k / experts : 1.0;
    double missed = 1.0;
    for (long long t = 0; t < r->tokens; ++t) missed *= 1.0 - hit;
    return (1.0 - missed) * experts * (double)tiles_per_expert <= 2.0 * sm_count();
}

}  // namespace

// Few rows per expert, on average.  SwiGLU and down product together, here against the kernel for many rows (us, L2 flushed):
// 32 experts, 2048 x 1408: 136 / 146 at 16 rows, 143 / 145 at 96, 159 / 150 at 128; 16 experts, 1024 x 2048: 68 / 78, 71 / 78,
// 82 / 80; 8 experts, 1024 x 2816: 60 / 68, 66 / 69, 66 / 70.  30 shapes of 4 .. 64 experts at 24 .. 96 rows: 0.65 .. 1.00 of the
// other's time under uniform load, and 0.70 .. 1.05 with lognormal load (sigma 1).  Two things lose:
//   * a few tiles with a long contraction each, whose time is what one SM can fetch: the other kernel splits a tile over two (8
//     experts, 2048 x 264, 24 tiles of gate and up: 39 / 41 at 24 rows, 41 / 39 at 96, with lognormal load 43 / 39; 960 x 320
//     35 / 37 at every count).  They change over at 24 rows.
//   * a load that has collapsed onto a few experts, which this side of the launch cannot see: all 6016 rows on one of 64
//     experts 125 / 98.
// The mean is of the whole route.  An expert-parallel view counts the tokens of all ranks over its own experts and so
// changes over earlier than it need, by the number of ranks.
constexpr long long kStreamRowsPerExpert = 96, kStreamRowsOfFewTiles = 24;
bool stream_down_early(const qmoe_route_t* r, const qmoe_experts_t* ex) { return few_tokens(r, ex->experts, ceil_div(ex->hidden, SM_ROWS)); }
bool stream_shape_ok(const qmoe_route_t* r, const qmoe_experts_t* ex) {
    const long long tiles = (long long)ex->experts * ceil_div(ex->hidden, SM_ROWS);
    const long long rows = tiles * 4 <= sm_count() && ex->width > 1536 ? kStreamRowsOfFewTiles : kStreamRowsPerExpert;
    return r->tokens * r->top_k <= rows * ex->experts && !kernel_variant(QMOE_VARIANT_NO_STREAM_GEMM);
}

int stream_swiglu_forward(const qmoe_route_t* r, const qmoe_experts_t* ex, uint64_t x, uint64_t g, uint64_t u, uint64_t h, bool pad_rows, bool early, bool let_next,
                          cudaStream_t stream) {
    StreamParams p = {};
    const uint64_t d = (uint64_t)ex->width, hd = (uint64_t)ex->hidden, E = (uint64_t)ex->experts;
    if (int rc = make_map_2d(&p.map_w, ex->w_gate, d, E * hd, SM_ROWS)) return rc;
    if (int rc = make_map_2d(&p.map_w2, ex->w_up, d, E * hd, SM_ROWS)) return rc;
    if (int rc = make_map_2d(&p.map_x, x, d, (uint64_t)r->rows_bound, X_BOX)) return rc;
    p.offsets = (const int*)r->offsets; p.counts = (const int*)r->counts; p.status = device_status_address();
    p.out0 = (__nv_bfloat16*)g; p.out1 = (__nv_bfloat16*)u; p.out2 = (__nv_bfloat16*)h;
    p.experts = ex->experts; p.m_tiles = ceil_div((long long)hd, SM_ROWS); p.N = (int)hd; p.K = (int)d;
    p.pad_rows = pad_rows; p.early = early; p.let_next = let_next;
    return few_tokens(r, ex->experts, p.m_tiles) ? stream_launch<STREAM_SWIGLU, true>(p, r, stream) : stream_launch<STREAM_SWIGLU>(p, r, stream);
}

int stream_rows_nt(const qmoe_route_t* r, int experts, uint64_t a, uint64_t b, uint64_t c, long long K, long long N, bool pad_rows, bool early,
                   cudaStream_t stream) {
    StreamParams p = {};
    if (int rc = make_map_2d(&p.map_w, b, (uint64_t)K, (uint64_t)experts * N, SM_ROWS)) return rc;
    p.map_w2 = p.map_w;
    if (int rc = make_map_2d(&p.map_x, a, (uint64_t)K, (uint64_t)r->rows_bound, X_BOX)) return rc;
    p.offsets = (const int*)r->offsets; p.counts = (const int*)r->counts; p.status = device_status_address();
    p.out0 = (__nv_bfloat16*)c;
    p.experts = experts; p.N = (int)N; p.K = (int)K; p.pad_rows = pad_rows; p.early = early;
    // Two weight tiles per stage where that leaves a tile for every SM and an expert's rows take more than one box of
    // activations: 64 experts, 94 rows on average, 1408 -> 2048 columns: 81 us with one, 74 with two; but 16 experts, 96 rows,
    // 2048 -> 1024 columns (64 tiles of 256): 27 with one, 32 with two.
    if (r->tokens * r->top_k > (long long)X_BOX * experts && (long long)ceil_div(N, 2 * SM_ROWS) * experts >= sm_count()) {
        p.m_tiles = ceil_div(N, 2 * SM_ROWS);
        return stream_launch<STREAM_NT2>(p, r, stream);
    }
    p.m_tiles = ceil_div(N, SM_ROWS);
    return few_tokens(r, experts, p.m_tiles) ? stream_launch<STREAM_NT, true>(p, r, stream) : stream_launch<STREAM_NT>(p, r, stream);
}

}  // namespace qmoe
