// Causal self-attention with grouped key/value heads, head width 64, bf16 in and out, on the tcgen05 tensor cores:
//     out[b, t, h, :] = sum_{s <= t} softmax_s(q[b, t, h, :] . k[b, s, g(h), :] / 8) v[b, s, g(h), :],  g(h) = h / (heads / kv_heads)
// forward (with the log-sum-exp of every row kept for the backward) and backward (dq, dk, dv).
// Upstream: `attention` src/qutai/lm/layers.py:119-130, kernels lm_attention_bf16_d64 / _dq / _dkv
// src/qutai/backends/cuda/lm.cu:91-285 (wmma), CPU statement src/qutai/backends/cpu_lm.py:141-201.  Like those kernels
// this never writes the time x time scores: keys and values stream through shared memory in blocks of 128 positions.
//
// Warp 0 of a CTA asks TMA for the tiles (3-D tensor maps [batch][time][heads * 64], so positions past the end of a sequence
// arrive as zeros and no tile reaches into the next sequence), warp 1 issues the MMAs (one elected thread), the row warps
// own one TMEM lane per thread.  Probabilities never pass through shared memory: the rows read the scores out of tensor
// memory and put P (dS), rounded to bf16, back there, where the next product takes it as its A operand.
//   forward, per item (sequence, head, block of 128 queries) and key block:  S = Q K^T -> rows: max, exp2, sum, P -> O += P V,
//   accumulated in tensor memory and rescaled there when a row's maximum has risen.
//   backward for dq, per item and key block as well:  S = Q K^T, dP = dO V^T -> rows: P = exp(S / 8 - lse), dS = P (dP - delta) -> dQ += dS K.
//   backward for dk, dv, per (sequence, key/value head, key block), over the query heads of the group and the query blocks
//   at or after it, everything transposed (lanes = key positions):  S^T = K Q^T, dP^T = V dO^T -> rows: P^T, dS^T ->
//   dV += P^T dO, dK += dS^T Q.
// The products of the next block are issued before the rows have finished with this one (S has a second buffer in the
// backward and is taken into registers at once in the forward).  What bounds them: the forward and dq the chain of a row warp (load, maximum,
// exponentials, store, barrier) beside the exponential unit, which alone is 1024 cycles per 128 x 128 block and SM; dk, dv the handshakes
// of an iteration between row warps, MMA warp and TMA (500 of 2650 cycles per block in waits; without exponentials, row
// values and the dV and dK products it still took 72 of its 97 us).
// 4 sequences x 2048 positions, 16 heads in 4 groups: forward and backward 606 -> 250 us against the form with P and dS in shared memory and
// one block in flight, 242 with O rescaled behind the exponentials and delta from coalesced loads; 3 x 1501 positions,
// forward: 72, 37 and 32.
// Every wait is bounded; on expiry the CTA records a code in the library's status word and leaves.
#include "common.cuh"
#include "tc_ptx.cuh"

namespace qmoe {
namespace {

constexpr int D = 64;                 // head width
constexpr int BLOCK = 128;            // query rows of a CTA = key positions of a block
constexpr int TILE_BYTES = BLOCK * D * 2;          // 16 KiB: 128 rows x 128 bytes
constexpr int THREADS = 192;              // forward, dq: TMA warp, MMA warp, four row warps
// Row warps per 32 rows of the dk, dv kernel, which share the columns of a block between them
constexpr int DKV_PARTS = 2, DKV_THREADS = 64 + 128 * DKV_PARTS;
constexpr float LOG2E = 1.4426950408889634f;
enum { STATUS_ATTENTION_WAIT = 301 };

struct alignas(64) AttentionParams {
    CUtensorMap map_q, map_k, map_v, map_do;     // 3-D [batch][time][heads * 64] bf16, boxes of 64 x 128 x 1
    CUtensorMap map_k2, map_v2;                  // the same tensors in boxes of 64 x 64 x 1 (dq kernel with key blocks of 64)
    const __nv_bfloat16* out_in;  // backward: the forward's output
    const __nv_bfloat16* grad_out;
    __nv_bfloat16* out;           // forward: out; backward for dq: dq; backward for dk, dv: dk
    __nv_bfloat16* out2;          // backward for dk, dv: dv
    float* lse;                   // [batch * time * heads]
    float* delta;                 // [batch * time * heads]  sum_j grad_out * out of every row
    int* status;
    int batch, time, heads, kv_heads;
    int split;                    // backward for dk, dv: CTAs per key block (cluster size)
};

__device__ __forceinline__ void tma_load_3d(const CUtensorMap* map, uint32_t dst, uint32_t bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float exp2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {      // like fmaxf: a number rather than a NaN
    float y;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}
// 32 accumulator columns of one row, scaled, as 64 bytes of bf16
__device__ __forceinline__ void store_row32(uint4* dst, const uint32_t* r, float scale) {
    auto two = [&](int c) { return pack2(__uint_as_float(r[c]) * scale, __uint_as_float(r[c + 1]) * scale); };
#pragma unroll
    for (int c = 0; c < 32; c += 8) dst[c / 8] = make_uint4(two(c), two(c + 2), two(c + 4), two(c + 6));
}
__device__ __forceinline__ void load_shared4(uint32_t at, float* v) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void load_cluster4(uint32_t at, float* v) {
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(at) : "memory");
}
// Where the 16 contraction elements [16 kk, 16 kk + 16) of a bf16 operand start that the rows wrote over the scores they had
// read: a thread keeps to its own COLS columns, P (or the only operand) in their first half, dS in their second
template <int COLS> __device__ __forceinline__ constexpr uint32_t p_column(int kk) { return (uint32_t)(kk * 16 / COLS * COLS + kk * 16 % COLS / 2); }

struct Wait {   // bounded waits of one thread; the first that runs out marks the CTA
    volatile int* abort_flag;
    int* status;
    __device__ __forceinline__ bool operator()(uint32_t bar, uint32_t parity) const {
        if (mbar_wait(bar, parity, abort_flag)) return true;
        if (!*abort_flag) { *abort_flag = 1; atomicExch(status, STATUS_ATTENTION_WAIT); }
        return false;
    }
    // the same for a whole warp: all lanes go on, or none does
    __device__ __forceinline__ bool all(uint32_t bar, uint32_t parity) const { return __all_sync(0xffffffffu, (*this)(bar, parity)); }
};

// a CTA that gave up leaves its copies and MMAs in flight a bounded time to land before its shared memory and TMEM go away
__device__ __forceinline__ void linger_after_abort(const volatile int* abort_flag) {
    if (!*abort_flag) return;
    const unsigned long long start = global_ns();
    while (global_ns() - start < 2000000ull) __nanosleep(1000);
}

// ------------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(THREADS, 2)
attention_forward_kernel(const __grid_constant__ AttentionParams p) {
    // No static shared memory and a 1 KiB-aligned dynamic block: 80 KiB of tiles and half of the tensor memory per CTA,
    // so two are resident per SM and one's exponentials run beside the other's waits.
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int blocks = (p.time + BLOCK - 1) / BLOCK;
    // heaviest query blocks first: the last block of a sequence has the most key blocks to walk
    const int heads_all = p.heads * p.batch;
    const int i = blocks - 1 - (int)(blockIdx.x / heads_all);
    const int h = (int)(blockIdx.x % heads_all) % p.heads, b = (int)(blockIdx.x % heads_all) / p.heads;
    const int g = h / (p.heads / p.kv_heads);
    const int n = i + 1;                       // key blocks 0 .. i
    const uint32_t base = smem_u32(smem_raw);
    const uint32_t q_tile = base, k_tile = base + TILE_BYTES, v_tile = k_tile + 2 * TILE_BYTES;
    const uint32_t bars = v_tile + 2 * TILE_BYTES;
    enum { Q_FULL = 0, K_FULL = 1, K_EMPTY = 3, V_FULL = 5, V_EMPTY = 7, S_FULL = 9, S_TAKEN = 10, P_FULL = 11, O_DONE = 12, BARS = 13 };
    auto bar = [&](int which) { return bars + 8u * which; };
    uint32_t& s_tmem_base = *reinterpret_cast<uint32_t*>(smem_raw + 5 * TILE_BYTES + 8 * BARS);
    volatile int& s_abort = *reinterpret_cast<volatile int*>(smem_raw + 5 * TILE_BYTES + 8 * BARS + 4);
    if (base & 1023u) {   // the operand tiles need the alignment the declaration asks for
        chain_wait();
        if (threadIdx.x == 0) atomicExch(p.status, STATUS_ATTENTION_WAIT + 1);
        return;
    }
    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int w = 0; w < BARS; ++w) mbar_init(bar(w), (w == S_TAKEN || w == P_FULL) ? 4 : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        prefetch_map(&p.map_q); prefetch_map(&p.map_k); prefetch_map(&p.map_v);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    chain_wait();
    chain_next();      // the tensor memory is this block's
    const uint32_t tmem = s_tmem_base;
    const uint32_t tmem_s = tmem, tmem_o = tmem + 128, tmem_p = tmem + 192;    // 128 + 64 + 64 (bf16 pairs) columns
    const Wait wait{&s_abort, p.status};

    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(bar(Q_FULL), TILE_BYTES);
            tma_load_3d(&p.map_q, q_tile, bar(Q_FULL), h * D, i * BLOCK, b);
            for (int j = 0; j < n && !s_abort; ++j) {
                const int st = j & 1;
                const uint32_t parity = ((uint32_t)(j >> 1) & 1u) ^ 1u;
                if (!wait(bar(K_EMPTY + st), parity)) break;
                mbar_expect_tx(bar(K_FULL + st), TILE_BYTES);
                tma_load_3d(&p.map_k, k_tile + st * TILE_BYTES, bar(K_FULL + st), g * D, j * BLOCK, b);
                if (!wait(bar(V_EMPTY + st), parity)) break;
                mbar_expect_tx(bar(V_FULL + st), TILE_BYTES);
                tma_load_3d(&p.map_v, v_tile + st * TILE_BYTES, bar(V_FULL + st), g * D, j * BLOCK, b);
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc_s = make_idesc<false, false, 128>(128), idesc_o = make_idesc<false, true, 128>(D);
        // S = Q K^T of key block j: both K-major, contraction over the 64 columns
        auto scores = [&](int j) {
            const int st = j & 1;
            if (!wait.all(bar(K_FULL + st), (uint32_t)(j >> 1) & 1u)) return false;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk)
                    umma_bf16(tmem_s, make_desc(q_tile + kk * 32, 16, 1024), make_desc(k_tile + st * TILE_BYTES + kk * 32, 16, 1024), idesc_s, kk ? 1u : 0u);
                umma_commit(bar(S_FULL));
                umma_commit(bar(K_EMPTY + st));
            }
            __syncwarp();
            return true;
        };
        bool ok = wait.all(bar(Q_FULL), 0) && scores(0);
        for (int j = 0; ok && j < n; ++j) {
            const int st = j & 1;
            // the scores of the next block as soon as the rows hold this block's in registers
            if (j + 1 < n) ok = wait.all(bar(S_TAKEN), (uint32_t)j & 1u) && scores(j + 1);
            if (ok) ok = wait.all(bar(V_FULL + st), (uint32_t)(j >> 1) & 1u);
            if (ok) ok = wait.all(bar(P_FULL), (uint32_t)j & 1u);
            if (!ok) break;
            tc_fence_after();
            // O += P V: P from tensor memory, V as it lies in memory (rows = key positions) is the MN-major operand:
            // 16 positions every 2 KiB
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < BLOCK / 16; ++kk)
                    umma_bf16_ts(tmem_o, tmem_p + kk * 8, make_desc(v_tile + st * TILE_BYTES + kk * 2048, 8192, 1024), idesc_o, (j | kk) ? 1u : 0u);
                umma_commit(bar(O_DONE));
                umma_commit(bar(V_EMPTY + st));
            }
            __syncwarp();
        }
        // the last commit has arrived before this CTA's shared memory can go to another one
        if (ok) wait.all(bar(V_EMPTY + ((n - 1) & 1)), (uint32_t)((n - 1) >> 1) & 1u);
    } else {
        const int quad = warp & 3, row = quad * 32 + lane;
        const int tq = i * BLOCK + row;                      // this thread's query position
        const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
        const float scale2 = 0.125f * LOG2E;                 // 1 / sqrt(64), in the exponent of 2
        const uint64_t scale_pair = pair2(scale2, scale2);
        float m = -INFINITY, l = 0.f;
        bool ok = true;
        for (int j = 0; ok && j < n; ++j) {
            ok = wait.all(bar(S_FULL), (uint32_t)j & 1u);
            if (!ok) break;
            tc_fence_after();
            uint32_t s[BLOCK];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(tmem_s + lane_base + c * 32, s + c * 32);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(S_TAKEN));
            if (j == i) {
#pragma unroll
                for (int c = 0; c < BLOCK; ++c)
                    if (c > row) s[c] = 0xff800000u;         // -inf
            }
            float peak4[4] = {__uint_as_float(s[0]), __uint_as_float(s[1]), __uint_as_float(s[2]), __uint_as_float(s[3])};
#pragma unroll
            for (int c = 4; c < BLOCK; c += 2) peak4[(c >> 1) & 3] = max3(peak4[(c >> 1) & 3], __uint_as_float(s[c]), __uint_as_float(s[c + 1]));
            const float peak = fmaxf(max3(peak4[0], peak4[1], peak4[2]), peak4[3]);
            // The base of the exponentials is the maximum so far.  (Letting it lag behind by up to 2^8 would leave O alone in
            // most blocks, but then the largest probability of a row is no longer an exact 1 in bf16: 2.05e-3 instead of
            // 1.74e-3 from the exact result for scores of standard deviation 4.)
            float alpha = 1.f;
            if (j == 0) {
                m = peak;
            } else {
                const float m_new = fmaxf(m, peak);
                alpha = exp2_fast((m - m_new) * scale2);
                m = m_new;
                l *= alpha;
            }
            // Subtract, then multiply: a single fma against m * scale2 saves an instruction, but that product is rounded, so the
            // largest probability becomes 2^(up to half an ulp of the base) instead of 1 (scores of 2e5: out 2.2e-3 instead of
            // 2.9e-5 from the exact result, and dq, whose terms cancel, 0.31 instead of 7e-3).
            const uint64_t minus_m = pair2(-m, -m);
            uint64_t total2[2] = {0, 0};
            uint32_t packed[BLOCK / 2];
#pragma unroll
            for (int c = 0; c < BLOCK; c += 2) {
                float x0, x1;
                unpair2(mul2(add2(pair2(__uint_as_float(s[c]), __uint_as_float(s[c + 1])), minus_m), scale_pair), x0, x1);
                const float p0 = exp2_fast(x0), p1 = exp2_fast(x1);
                total2[(c >> 1) & 1] = add2(total2[(c >> 1) & 1], pair2(p0, p1));
                packed[c >> 1] = pack2(p0, p1);
            }
            if (j > 0) {
                // the product that reads the P of the block before is done: O is whole, and the place of P free.  Only here, behind
                // the exponentials: their registers are free for O by now, and the wait is over before it begins (before them, with
                // 16 columns at a time, wait and rescaling took 900 of a block's 3400 cycles)
                ok = wait.all(bar(O_DONE), (uint32_t)(j - 1) & 1u);
                if (!ok) break;
                tc_fence_after();
                if (__any_sync(0xffffffffu, alpha != 1.f)) {
                    uint32_t o[D];
                    tmem_ld32(tmem_o + lane_base, o);
                    tmem_ld32(tmem_o + lane_base + 32, o + 32);
                    tmem_ld_wait();
                    const uint64_t alpha_pair = pair2(alpha, alpha);
#pragma unroll
                    for (int e = 0; e < D; e += 2) {
                        float o0, o1;
                        unpair2(mul2(pair2(__uint_as_float(o[e]), __uint_as_float(o[e + 1])), alpha_pair), o0, o1);
                        o[e] = __float_as_uint(o0);
                        o[e + 1] = __float_as_uint(o1);
                    }
                    tmem_st32(tmem_o + lane_base, o);
                    tmem_st32(tmem_o + lane_base + 32, o + 32);
                }
            }
            tmem_st32(tmem_p + lane_base, packed);
            tmem_st32(tmem_p + lane_base + 32, packed + 32);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(P_FULL));
            float t0, t1;
            unpair2(add2(total2[0], total2[1]), t0, t1);
            l += t0 + t1;
        }
        if (ok) ok = wait.all(bar(O_DONE), (uint32_t)(n - 1) & 1u);
        if (ok) {
            tc_fence_after();
            uint32_t o[D];
            tmem_ld32(tmem_o + lane_base, o);
            tmem_ld32(tmem_o + lane_base + 32, o + 32);
            tmem_ld_wait();
            if (tq < p.time) {
                const float inverse = 1.f / l;
                const long long at = ((long long)b * p.time + tq) * p.heads + h;
                uint4* dst = reinterpret_cast<uint4*>(p.out + at * D);
                auto value = [&](int c) { return __uint_as_float(o[c]) * inverse; };
#pragma unroll
                for (int c = 0; c < D; c += 8)
                    dst[c / 8] = make_uint4(pack2(value(c), value(c + 1)), pack2(value(c + 2), value(c + 3)),
                                            pack2(value(c + 4), value(c + 5)), pack2(value(c + 6), value(c + 7)));
                p.lse[at] = m * 0.125f + __logf(l);
            }
        }
    }
    linger_after_abort(&s_abort);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
    }
}


// ------------------------------------------------------------------------------------------------
// backward, part 1: dq (and delta), one CTA per (sequence, head, query block); key blocks of 64 positions.  A CTA needs
// 256 TMEM columns (two S, one dP, dQ) and 80 KiB, so two are resident per SM.
// ------------------------------------------------------------------------------------------------
constexpr int DQ_KV = 64, DQ_TILE = DQ_KV * 128, DQ_STAGES = 3;
constexpr int DQ_TILES = 2 * TILE_BYTES + 2 * DQ_STAGES * DQ_TILE;
constexpr int DQ_SMEM = DQ_TILES + 128;

__global__ void __launch_bounds__(THREADS, 2)
attention_dq_kernel(const __grid_constant__ AttentionParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int blocks = (p.time + BLOCK - 1) / BLOCK;
    const int heads_all = p.heads * p.batch;
    const int i = blocks - 1 - (int)(blockIdx.x / heads_all);
    const int h = (int)(blockIdx.x % heads_all) % p.heads, b = (int)(blockIdx.x % heads_all) / p.heads;
    const int g = h / (p.heads / p.kv_heads);
    const int n = (i + 1) * (BLOCK / DQ_KV);   // key blocks that hold a position <= the last query of this block
    const uint32_t base = smem_u32(smem_raw);
    const uint32_t q_tile = base, do_tile = base + TILE_BYTES, k_tile = do_tile + TILE_BYTES, v_tile = k_tile + DQ_STAGES * DQ_TILE;
    const uint32_t bars = base + DQ_TILES;
    enum { Q_FULL = 0, KV_FULL = 1, KV_EMPTY = KV_FULL + DQ_STAGES, S_FULL = KV_EMPTY + DQ_STAGES, DP_FULL = S_FULL + 2, DS_FULL, DQ_DONE, BARS };
    auto bar = [&](int which) { return bars + 8u * which; };
    uint32_t& s_tmem_base = *reinterpret_cast<uint32_t*>(smem_raw + DQ_TILES + 8 * BARS);
    volatile int& s_abort = *reinterpret_cast<volatile int*>(smem_raw + DQ_TILES + 8 * BARS + 4);
    if (base & 1023u) {
        chain_wait();
        if (threadIdx.x == 0) atomicExch(p.status, STATUS_ATTENTION_WAIT + 1);
        return;
    }
    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int w = 0; w < BARS; ++w) mbar_init(bar(w), w == DS_FULL ? 4 : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        prefetch_map(&p.map_q); prefetch_map(&p.map_k2); prefetch_map(&p.map_v2); prefetch_map(&p.map_do);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    chain_wait();
    chain_next();      // the tensor memory is this block's
    const uint32_t tmem = s_tmem_base;
    // S of block j in columns 64 (j & 1) ..; the rows put dS (bf16 pairs) back over the columns they read
    const uint32_t tmem_dp = tmem + 2 * DQ_KV, tmem_dq = tmem + 3 * DQ_KV;
    const Wait wait{&s_abort, p.status};

    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(bar(Q_FULL), 2 * TILE_BYTES);
            tma_load_3d(&p.map_q, q_tile, bar(Q_FULL), h * D, i * BLOCK, b);
            tma_load_3d(&p.map_do, do_tile, bar(Q_FULL), h * D, i * BLOCK, b);
            int st = 0;
            uint32_t parity = 1;
            for (int j = 0; j < n && !s_abort; ++j) {
                if (!wait(bar(KV_EMPTY + st), parity)) break;
                mbar_expect_tx(bar(KV_FULL + st), 2 * DQ_TILE);
                tma_load_3d(&p.map_k2, k_tile + st * DQ_TILE, bar(KV_FULL + st), g * D, j * DQ_KV, b);
                tma_load_3d(&p.map_v2, v_tile + st * DQ_TILE, bar(KV_FULL + st), g * D, j * DQ_KV, b);
                if (++st == DQ_STAGES) { st = 0; parity ^= 1u; }
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc_s = make_idesc<false, false, 128>(DQ_KV), idesc_dq = make_idesc<false, true, 128>(D);
        // S = Q K^T of block j into its buffer
        auto scores = [&](int j) {
            const int st = j % DQ_STAGES;
            if (!wait.all(bar(KV_FULL + st), (uint32_t)(j / DQ_STAGES) & 1u)) return false;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk)
                    umma_bf16(tmem + (uint32_t)(j & 1) * DQ_KV, make_desc(q_tile + kk * 32, 16, 1024),
                              make_desc(k_tile + st * DQ_TILE + kk * 32, 16, 1024), idesc_s, kk ? 1u : 0u);
                umma_commit(bar(S_FULL + (j & 1)));
            }
            __syncwarp();
            return true;
        };
        auto d_probabilities = [&](int j) {    // dP = dO V^T of block j
            const int st = j % DQ_STAGES;
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk)
                    umma_bf16(tmem_dp, make_desc(do_tile + kk * 32, 16, 1024), make_desc(v_tile + st * DQ_TILE + kk * 32, 16, 1024), idesc_s, kk ? 1u : 0u);
                umma_commit(bar(DP_FULL));
            }
            __syncwarp();
        };
        bool ok = wait.all(bar(Q_FULL), 0) && scores(0);
        if (ok) d_probabilities(0);
        for (int j = 0; ok && j < n; ++j) {
            // the scores of the next block into the other buffer, once the product that reads the dS of block j - 1 there is done
            if (j > 0) ok = wait.all(bar(KV_EMPTY + (j - 1) % DQ_STAGES), (uint32_t)((j - 1) / DQ_STAGES) & 1u);
            if (ok && j + 1 < n) ok = scores(j + 1);
            if (ok) ok = wait.all(bar(DS_FULL), (uint32_t)j & 1u);
            if (!ok) break;
            tc_fence_after();
            if (j + 1 < n) d_probabilities(j + 1);       // the rows have read this block's dP
            const int st = j % DQ_STAGES;
            // dQ += dS K: dS from tensor memory, the K tile read as the MN-major operand (rows = key positions)
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < DQ_KV / 16; ++kk)
                    umma_bf16_ts(tmem_dq, tmem + (uint32_t)(j & 1) * DQ_KV + p_column<DQ_KV>(kk),
                                 make_desc(k_tile + st * DQ_TILE + kk * 2048, 8192, 1024), idesc_dq, (j | kk) ? 1u : 0u);
                umma_commit(bar(KV_EMPTY + st));
                if (j == n - 1) umma_commit(bar(DQ_DONE));
            }
            __syncwarp();
        }
        if (ok) wait.all(bar(DQ_DONE), 0);         // the last commit has arrived
    } else {
        constexpr int COLS = DQ_KV;                // columns of a block per thread
        const int quad = warp & 3, row = quad * 32 + lane;
        const int tq = i * BLOCK + row;
        const bool live = tq < p.time;
        const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
        const long long at = ((long long)b * p.time + (live ? tq : 0)) * p.heads + h;
        // delta = sum_j grad_out * out of this row (kept for the dk, dv kernel), lse of this row.  Eight lanes read a row, four rows
        // per access, and all accesses are on their way before the first sum (a row per lane, 16 bytes at a time: 3 us of
        // the 10 .. 30 of a CTA before its first block).  The pairs of a row are added in their order, from lane to lane, as one thread
        // per row would add them: the order is part of the result (4 sequences x 2048 positions, 16 heads, this
        // kernel alone: 78 us with a row per thread, 75 like this; each lane's eight products summed first would save another 1 us).
        float delta = 0.f, lse2 = 0.f;
        {
            uint4 a[8], o[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int t = i * BLOCK + quad * 32 + r * 4 + (lane >> 3);
                const long long from = (((long long)b * p.time + (t < p.time ? t : 0)) * p.heads + h) * (D / 8) + (lane & 7);
                a[r] = reinterpret_cast<const uint4*>(p.grad_out)[from];
                o[r] = reinterpret_cast<const uint4*>(p.out_in)[from];
            }
            if (live) lse2 = p.lse[at] * LOG2E;
            float pairs[8][4], sum[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const uint32_t aw[4] = {a[r].x, a[r].y, a[r].z, a[r].w}, ow[4] = {o[r].x, o[r].y, o[r].z, o[r].w};
                sum[r] = 0.f;
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    pairs[r][e] = __uint_as_float(aw[e] << 16) * __uint_as_float(ow[e] << 16) +
                                  __uint_as_float(aw[e] & 0xffff0000u) * __uint_as_float(ow[e] & 0xffff0000u);
            }
#pragma unroll 1
            for (int c = 0; c < D / 8; ++c) {
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    float s = sum[r];
#pragma unroll
                    for (int e = 0; e < 4; ++e) s += pairs[r][e];
                    sum[r] = __shfl_sync(0xffffffffu, s, c, 8);      // of the lane that holds this piece of the row
                }
            }
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float mine = __shfl_sync(0xffffffffu, sum[r], (lane & 3) * 8);      // of row 4 r + (lane & 3)
                if ((lane >> 2) == r) delta = mine;
            }
            if (live) p.delta[at] = delta;
            else delta = 0.f;
        }
        const float scale2 = 0.125f * LOG2E;
        const uint64_t scale_pair = pair2(scale2, scale2), lse_pair = pair2(-lse2, -lse2), delta_pair = pair2(-delta, -delta);
        bool ok = true;
        for (int j = 0; ok && j < n; ++j) {
            const uint32_t tmem_s = tmem + (uint32_t)(j & 1) * DQ_KV + lane_base;
            const int first = j * DQ_KV - i * BLOCK;                     // first key position of the block, from the CTA's first query
            const bool masked = first + COLS - 1 > quad * 32;            // some row of this warp may not see some of these columns
            uint32_t s[COLS], dp[COLS], packed[COLS / 2];
            ok = wait.all(bar(S_FULL + (j & 1)), (uint32_t)(j >> 1) & 1u);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < COLS; c += 32) tmem_ld32(tmem_s + c, s + c);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < COLS; c += 2) {
                float x0, x1;
                unpair2(fma2(pair2(__uint_as_float(s[c]), __uint_as_float(s[c + 1])), scale_pair, lse_pair), x0, x1);
                s[c] = __float_as_uint(exp2_fast(x0));
                s[c + 1] = __float_as_uint(exp2_fast(x1));
            }
            ok = wait.all(bar(DP_FULL), (uint32_t)j & 1u);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < COLS; c += 32) tmem_ld32(tmem_dp + lane_base + c, dp + c);
            tmem_ld_wait();
            // dS without the 1/8 of the scores, which the last step applies to dQ (a power of two: the same bits)
#pragma unroll
            for (int c = 0; c < COLS; c += 2) {
                float d0, d1;
                unpair2(mul2(pair2(__uint_as_float(s[c]), __uint_as_float(s[c + 1])),
                             add2(pair2(__uint_as_float(dp[c]), __uint_as_float(dp[c + 1])), delta_pair)), d0, d1);
                s[c] = __float_as_uint(d0);
                s[c + 1] = __float_as_uint(d1);
            }
            if (masked) {      // a loop of its own: as selects in the one above the mask cost every block, not only those on the diagonal
#pragma unroll
                for (int c = 0; c < COLS; ++c)
                    if (first + c > row) s[c] = 0u;
            }
#pragma unroll
            for (int c = 0; c < COLS; c += 2) packed[c >> 1] = pack2(__uint_as_float(s[c]), __uint_as_float(s[c + 1]));
            tmem_st32(tmem_s, packed);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(DS_FULL));
        }
        if (ok) ok = wait.all(bar(DQ_DONE), 0);
        if (ok) {
            tc_fence_after();
            uint4* dst = reinterpret_cast<uint4*>(p.out + at * D);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t r[32];
                tmem_ld32(tmem_dq + lane_base + c * 32, r);
                tmem_ld_wait();
                if (live) store_row32(dst + c * 4, r, 0.125f);
            }
        }
    }
    linger_after_abort(&s_abort);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------
// backward, part 2: dk and dv, one CTA per (sequence, key/value head, key block) and, where those are too few to fill the
// machine, a cluster of `p.split` CTAs that share its (query head, query block) list and add their dk, dv through
// distributed shared memory in a fixed order.
// ------------------------------------------------------------------------------------------------
constexpr int DKV_STAGES = 3;
constexpr int DKV_ROW_BYTES = 2 * BLOCK * 4;          // -lse * log2 e and -delta of a query block
constexpr int DKV_TILES = (2 + 2 * DKV_STAGES) * TILE_BYTES;
constexpr int DKV_SUM_PITCH = 128 * 4 + 16;            // one row of dv and dk sums; 16 more bytes spread the rows over the banks
static_assert(BLOCK * DKV_SUM_PITCH <= 2 * DKV_STAGES * TILE_BYTES, "the sums fit where the query tiles were");
constexpr int DKV_SMEM = DKV_TILES + DKV_STAGES * DKV_ROW_BYTES + 128;

__global__ void __launch_bounds__(DKV_THREADS, 1)
attention_dkv_kernel(const __grid_constant__ AttentionParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int blocks = (p.time + BLOCK - 1) / BLOCK;
    const int heads_all = p.kv_heads * p.batch, job = (int)blockIdx.x / p.split, share = (int)blockIdx.x % p.split;
    const int j = job / heads_all;                             // the first key block has the most query blocks to walk
    const int g = job % heads_all % p.kv_heads, b = job % heads_all / p.kv_heads;
    const int group = p.heads / p.kv_heads;
    const int per_head = blocks - j;                           // query blocks j .. blocks - 1
    const int all = group * per_head;                          // iterations: head of the group (outer), query block (inner)
    const int begin = all * share / p.split, n = all * (share + 1) / p.split - begin;      // this CTA's (none, when there are fewer than CTAs)
    const int first_head = begin / per_head, first_i = j + begin % per_head;
    const uint32_t base = smem_u32(smem_raw);
    const uint32_t k_tile = base, v_tile = base + TILE_BYTES, q_tile = v_tile + TILE_BYTES, do_tile = q_tile + DKV_STAGES * TILE_BYTES;
    const uint32_t rows_at = base + DKV_TILES, bars = rows_at + DKV_STAGES * DKV_ROW_BYTES;
    enum { KV_FULL = 0, Q_FULL = 1, Q_EMPTY = Q_FULL + DKV_STAGES, S_FULL = Q_EMPTY + DKV_STAGES, DP_FULL = S_FULL + 2, P_FULL, DS_FULL = P_FULL + 2, ACC_DONE, BARS };
    // S_FULL and P_FULL are two barriers each, by the parity of the iteration: the scores of the next iteration are formed before
    // all rows have put back this one's P, so a fast warp may be a whole phase ahead of a slow one there, and with one barrier
    // its second arrival would stand in for the slow warp's first.  (DS_FULL: the next dP waits for this phase.)
    auto bar = [&](int which) { return bars + 8u * which; };
    uint32_t& s_tmem_base = *reinterpret_cast<uint32_t*>(smem_raw + DKV_TILES + DKV_STAGES * DKV_ROW_BYTES + 8 * BARS);
    volatile int& s_abort = *reinterpret_cast<volatile int*>(smem_raw + DKV_TILES + DKV_STAGES * DKV_ROW_BYTES + 8 * BARS + 4);
    if (base & 1023u) {
        chain_wait();
        if (threadIdx.x == 0) atomicExch(p.status, STATUS_ATTENTION_WAIT + 1);
        return;
    }
    if (threadIdx.x == 0) {
        s_abort = 0;
        // a stage is full when its bytes have landed and the lanes of the loading warp have written its row values
        for (int w = 0; w < BARS; ++w) {
            const bool rows = w >= P_FULL && w <= DS_FULL, full = w >= Q_FULL && w < Q_EMPTY;
            mbar_init(bar(w), rows ? 4 * DKV_PARTS : full ? 2 : 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        prefetch_map(&p.map_q); prefetch_map(&p.map_k); prefetch_map(&p.map_v); prefetch_map(&p.map_do);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    chain_wait();
    chain_next();      // the tensor memory is this block's
    const uint32_t tmem = s_tmem_base;
    // everything with key positions as rows (lanes) and query positions as columns: S^T of iteration it in columns
    // 128 (it & 1) .., over which the rows put back P^T and dS^T (bf16 pairs); one dP^T
    const uint32_t tmem_dp = tmem + 256, tmem_dv = tmem + 384, tmem_dk = tmem + 448;
    const Wait wait{&s_abort, p.status};

    if (n == 0) {
        // nothing to do before the sum
    } else if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(bar(KV_FULL), 2 * TILE_BYTES);
            tma_load_3d(&p.map_k, k_tile, bar(KV_FULL), g * D, j * BLOCK, b);
            tma_load_3d(&p.map_v, v_tile, bar(KV_FULL), g * D, j * BLOCK, b);
        }
        int st = 0, head = first_head, i = first_i;
        uint32_t parity = 1;
        bool ok = true;
        for (int it = 0; ok && it < n; ++it) {
            const int h = g * group + head;
            // the row values travel through registers while the stage is still in use
            float lse2[BLOCK / 32], delta[BLOCK / 32];
#pragma unroll
            for (int r = 0; r < BLOCK / 32; ++r) {
                const int tq = i * BLOCK + r * 32 + lane;
                const long long at = ((long long)b * p.time + tq) * p.heads + h;
                const bool live = tq < p.time;                       // past the end: a probability of zero
                lse2[r] = live ? -p.lse[at] * LOG2E : -INFINITY;
                delta[r] = live ? -p.delta[at] : 0.f;
            }
            ok = wait.all(bar(Q_EMPTY + st), parity);
            if (!ok) break;
            if (lane == 0) {
                mbar_expect_tx(bar(Q_FULL + st), 2 * TILE_BYTES);
                tma_load_3d(&p.map_q, q_tile + st * TILE_BYTES, bar(Q_FULL + st), h * D, i * BLOCK, b);
                tma_load_3d(&p.map_do, do_tile + st * TILE_BYTES, bar(Q_FULL + st), h * D, i * BLOCK, b);
            }
            float* rows = reinterpret_cast<float*>(smem_raw + DKV_TILES + st * DKV_ROW_BYTES);
#pragma unroll
            for (int r = 0; r < BLOCK / 32; ++r) {
                rows[r * 32 + lane] = lse2[r];
                rows[BLOCK + r * 32 + lane] = delta[r];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(Q_FULL + st));
            if (++st == DKV_STAGES) { st = 0; parity ^= 1u; }
            if (++i == blocks) { i = j; ++head; }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc_s = make_idesc<false, false, 128>(128), idesc_t = make_idesc<false, true, 128>(D);
        auto scores = [&](int it) {      // S^T = K Q^T
            const int st = it % DKV_STAGES;
            if (!wait.all(bar(Q_FULL + st), (uint32_t)(it / DKV_STAGES) & 1u)) return false;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk)
                    umma_bf16(tmem + (uint32_t)(it & 1) * 128, make_desc(k_tile + kk * 32, 16, 1024),
                              make_desc(q_tile + st * TILE_BYTES + kk * 32, 16, 1024), idesc_s, kk ? 1u : 0u);
                umma_commit(bar(S_FULL + (it & 1)));
            }
            __syncwarp();
            return true;
        };
        auto d_probabilities = [&](int it) {    // dP^T = V dO^T
            const int st = it % DKV_STAGES;
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk)
                    umma_bf16(tmem_dp, make_desc(v_tile + kk * 32, 16, 1024), make_desc(do_tile + st * TILE_BYTES + kk * 32, 16, 1024), idesc_s, kk ? 1u : 0u);
                umma_commit(bar(DP_FULL));
            }
            __syncwarp();
        };
        bool ok = wait.all(bar(KV_FULL), 0) && scores(0);
        if (ok) d_probabilities(0);
        for (int it = 0; ok && it < n; ++it) {
            const int st = it % DKV_STAGES;
            const uint32_t buffer = tmem + (uint32_t)(it & 1) * 128;
            // the next scores into the other buffer, once the products that read the P and dS of iteration it - 1 there are done
            if (it > 0) ok = wait.all(bar(Q_EMPTY + (it - 1) % DKV_STAGES), (uint32_t)((it - 1) / DKV_STAGES) & 1u);
            if (ok && it + 1 < n) ok = scores(it + 1);
            if (ok) ok = wait.all(bar(P_FULL + (it & 1)), (uint32_t)(it >> 1) & 1u);
            if (!ok) break;
            tc_fence_after();
            // dV += P^T dO and dK += dS^T Q: P^T and dS^T from tensor memory, dO and Q as they lie in memory (rows = query
            // positions = the contraction) are MN-major operands
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < BLOCK / 16; ++kk)
                    umma_bf16_ts(tmem_dv, buffer + p_column<BLOCK / DKV_PARTS>(kk), make_desc(do_tile + st * TILE_BYTES + kk * 2048, 8192, 1024),
                                 idesc_t, (it | kk) ? 1u : 0u);
            }
            __syncwarp();
            ok = wait.all(bar(DS_FULL), (uint32_t)it & 1u);
            if (!ok) break;
            tc_fence_after();
            if (it + 1 < n) d_probabilities(it + 1);     // the rows have read this iteration's dP
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < BLOCK / 16; ++kk)
                    umma_bf16_ts(tmem_dk, buffer + p_column<BLOCK / DKV_PARTS>(kk) + BLOCK / DKV_PARTS / 2,
                                 make_desc(q_tile + st * TILE_BYTES + kk * 2048, 8192, 1024), idesc_t, (it | kk) ? 1u : 0u);
                umma_commit(bar(Q_EMPTY + st));
                if (it == n - 1) umma_commit(bar(ACC_DONE));
            }
            __syncwarp();
        }
        if (ok) wait.all(bar(ACC_DONE), 0);        // the last commit has arrived
    } else {
        constexpr int COLS = BLOCK / DKV_PARTS;    // columns (query positions) of a block per thread
        const int quad = warp & 3, row = quad * 32 + lane, part = (warp - 2) >> 2;
        const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
        const float scale2 = 0.125f * LOG2E;
        const uint64_t scale_pair = pair2(scale2, scale2);
        int st = 0, i = first_i;
        bool ok = true;
        for (int it = 0; ok && it < n; ++it) {
            const uint32_t tmem_s = tmem + (uint32_t)(it & 1) * 128 + lane_base + part * COLS;
            const uint32_t row_values = rows_at + st * DKV_ROW_BYTES + part * COLS * 4;
            const bool masked = i == j && part * COLS < quad * 32 + 31;  // some row of this warp is not seen by some of these columns
            const int live = p.time - i * BLOCK - part * COLS;           // columns from here on are past the end of the sequence
            uint32_t s[COLS], dp[COLS];
            auto put_back = [&](uint32_t to) {         // s, rounded to bf16, 32 columns at a time (the registers of all at once spill)
#pragma unroll
                for (int c = 0; c < COLS; c += 32) {
                    uint32_t packed[16];
#pragma unroll
                    for (int e = 0; e < 32; e += 2) packed[e >> 1] = pack2(__uint_as_float(s[c + e]), __uint_as_float(s[c + e + 1]));
                    tmem_st16(to + c / 2, packed);
                }
            };
            // the row values of this stage (the scores of this iteration were formed from the same stage, but the barrier that
            // publishes the loading warp's plain stores is the stage's own)
            ok = wait.all(bar(Q_FULL + st), (uint32_t)(it / DKV_STAGES) & 1u);
            if (ok) ok = wait.all(bar(S_FULL + (it & 1)), (uint32_t)(it >> 1) & 1u);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < COLS; c += 32) tmem_ld32(tmem_s + c, s + c);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < COLS; c += 4) {
                float l[4], x[4];
                load_shared4(row_values + c * 4, l);
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    unpair2(fma2(pair2(__uint_as_float(s[c + e]), __uint_as_float(s[c + e + 1])), scale_pair, pair2(l[e], l[e + 1])), x[e], x[e + 1]);
                    s[c + e] = __float_as_uint(exp2_fast(x[e]));
                    s[c + e + 1] = __float_as_uint(exp2_fast(x[e + 1]));
                }
            }
            if (masked) {      // a loop of its own, as in the dq kernel (both: 191 -> 181 us at 4 x 2048 positions, 16 heads)
#pragma unroll
                for (int c = 0; c < COLS; ++c)
                    if (part * COLS + c < row) s[c] = 0u;
            }
            if (live < COLS) {     // their scores are 0 * key: NaN for a key with an infinite component, although nobody sees it
#pragma unroll
                for (int c = 0; c < COLS; ++c)
                    if (c >= live) s[c] = 0u;
            }
            put_back(tmem_s);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(P_FULL + (it & 1)));
            ok = wait.all(bar(DP_FULL), (uint32_t)it & 1u);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < COLS; c += 32) tmem_ld32(tmem_dp + lane_base + part * COLS + c, dp + c);
            tmem_ld_wait();
            // dS without the 1/8 of the scores, which the last step applies to dK (a power of two: the same bits)
#pragma unroll
            for (int c = 0; c < COLS; c += 4) {
                float d[4];
                load_shared4(row_values + BLOCK * 4 + c * 4, d);
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    float d0, d1;
                    unpair2(mul2(pair2(__uint_as_float(s[c + e]), __uint_as_float(s[c + e + 1])),
                                 add2(pair2(__uint_as_float(dp[c + e]), __uint_as_float(dp[c + e + 1])), pair2(d[e], d[e + 1]))), d0, d1);
                    s[c + e] = __float_as_uint(d0);
                    s[c + e + 1] = __float_as_uint(d1);
                }
            }
            if (masked) {
#pragma unroll
                for (int c = 0; c < COLS; ++c)
                    if (part * COLS + c < row) s[c] = 0u;
            }
            put_back(tmem_s + COLS / 2);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(DS_FULL));
            if (++st == DKV_STAGES) st = 0;
            if (++i == blocks) i = j;
        }
        if (ok) ok = wait.all(bar(ACC_DONE), 0);
        if (ok) {
            tc_fence_after();
            const int tk = j * BLOCK + row;                     // this thread's key position
            const long long at = ((long long)b * p.time + (tk < p.time ? tk : 0)) * p.kv_heads + g;
#pragma unroll
            for (int c = part; c < 4; c += DKV_PARTS) {         // 32-column chunks 0, 1: dv; 2, 3: dk
                uint32_t r[32];
                tmem_ld32(tmem_dv + lane_base + c * 32, r);
                tmem_ld_wait();
                if (p.split > 1) {      // the tiles of this CTA are spent: its sums take their place
                    float4* sums = reinterpret_cast<float4*>(smem_raw + 2 * TILE_BYTES + row * DKV_SUM_PITCH + c * 128);
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        sums[e] = make_float4(__uint_as_float(r[4 * e]), __uint_as_float(r[4 * e + 1]), __uint_as_float(r[4 * e + 2]), __uint_as_float(r[4 * e + 3]));
                } else if (tk < p.time) {
                    store_row32(reinterpret_cast<uint4*>((c >> 1 ? p.out : p.out2) + at * D) + (c & 1) * 4, r, c >> 1 ? 0.125f : 1.f);
                }
            }
        }
    }
    linger_after_abort(&s_abort);
    tc_fence_before();
    if (p.split > 1) {
        cluster_sync();
        // every CTA adds the sums of all for its share of the 128 rows: 16 pieces of 8 columns (0-7: dv, 8-15: dk) per row
        const int row0 = BLOCK * share / p.split, rows = BLOCK * (share + 1) / p.split - row0;
        for (int at = threadIdx.x; at < rows * 16; at += DKV_THREADS) {
            const int row = row0 + at / 16, piece = at % 16, tk = j * BLOCK + row;
            float total[8] = {};
            for (int other = 0; other < p.split; ++other) {
                if (all * (other + 1) / p.split == all * other / p.split) continue;        // had no iterations
                const uint32_t from = map_to_cta(q_tile + row * DKV_SUM_PITCH + piece * 32, other);
                float v[8];
                load_cluster4(from, v);
                load_cluster4(from + 16, v + 4);
#pragma unroll
                for (int e = 0; e < 8; ++e) total[e] += v[e];
            }
            const float scale = piece >> 3 ? 0.125f : 1.f;
            if (tk < p.time)
                reinterpret_cast<uint4*>((piece >> 3 ? p.out : p.out2) + (((long long)b * p.time + tk) * p.kv_heads + g) * D)[piece & 7] =
                    make_uint4(pack2(total[0] * scale, total[1] * scale), pack2(total[2] * scale, total[3] * scale),
                               pack2(total[4] * scale, total[5] * scale), pack2(total[6] * scale, total[7] * scale));
        }
        cluster_sync();        // nobody leaves while its sums are being read
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

constexpr int FORWARD_SMEM = 5 * TILE_BYTES + 128;

}  // namespace

// CTAs per key block of the dk, dv kernel: one while the longest list (the first key block's: every query block of every
// head of the group) is within a quarter of the SMs' average share, else as many, up to 8 and a power of two, as bring it there.
int dkv_split(const qmoe_attention_t* a, int blocks) {
    const long long group = a->heads / a->kv_heads, longest = group * blocks;
    const long long total = (long long)a->batch * a->kv_heads * group * blocks * (blocks + 1) / 2, share = total / sm_count();
    int split = 1;
    while (split < 8 && longest * 4 > (share * 5 + 4) * split && longest > 2 * split) split *= 2;
    return split;
}

int attention_check(const qmoe_attention_t* a, bool backward) {
    if (!a) return fail_arg("attention is null");
    if (a->dim != D) return fail_arg("attention: head width must be 64");
    if (a->dtype != QMOE_BF16) return fail_arg("attention: dtype must be QMOE_BF16");
    if (a->batch <= 0 || a->time <= 0 || a->heads <= 0 || a->kv_heads <= 0 || a->heads % a->kv_heads)
        return fail_arg("attention: sizes must be positive and heads a multiple of kv_heads");
    if ((long long)a->batch * a->time * a->heads * D > (1ll << 40)) return fail_arg("attention: too large");
    if (!a->q || !a->k || !a->v || !a->out || !a->lse) return fail_arg("attention: null buffer address");
    if (backward && (!a->grad_out || !a->delta || !a->dq || !a->dk || !a->dv)) return fail_arg("attention_backward: null buffer address");
    if ((a->q | a->k | a->v | a->out | a->grad_out | a->dq | a->dk | a->dv) & 15u) return fail_arg("attention: buffers must be 16-byte aligned");
    return 0;
}

}  // namespace qmoe

using namespace qmoe;

extern "C" int qmoe_attention_forward(const qmoe_attention_t* a, uint64_t stream_) {
    if (int rc = attention_check(a, false)) return rc;
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_ATTENTION, stream);
    AttentionParams p = {};
    const uint64_t wide = (uint64_t)a->heads * D, narrow = (uint64_t)a->kv_heads * D;
    if (int rc = make_map_3d(&p.map_q, a->q, wide, (uint64_t)a->time, (uint64_t)a->batch, BLOCK)) return rc;
    if (int rc = make_map_3d(&p.map_k, a->k, narrow, (uint64_t)a->time, (uint64_t)a->batch, BLOCK)) return rc;
    if (int rc = make_map_3d(&p.map_v, a->v, narrow, (uint64_t)a->time, (uint64_t)a->batch, BLOCK)) return rc;
    p.out = (__nv_bfloat16*)a->out; p.lse = (float*)a->lse; p.status = device_status_address();
    p.batch = a->batch; p.time = a->time; p.heads = a->heads; p.kv_heads = a->kv_heads;
    QMOE_CUDA(cudaFuncSetAttribute(attention_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FORWARD_SMEM));
    const int blocks = (a->time + BLOCK - 1) / BLOCK;
    chained(attention_forward_kernel, (unsigned)(blocks * a->heads * a->batch), THREADS, FORWARD_SMEM, stream, p);
    count_tensor_core_launch();
    QMOE_LAUNCH_CHECK("attention_forward_kernel");
    return 0;
}

extern "C" int qmoe_attention_backward(const qmoe_attention_t* a, uint64_t stream_) {
    if (int rc = attention_check(a, true)) return rc;
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_ATTENTION, stream);
    AttentionParams p = {};
    const uint64_t wide = (uint64_t)a->heads * D, narrow = (uint64_t)a->kv_heads * D;
    if (int rc = make_map_3d(&p.map_q, a->q, wide, (uint64_t)a->time, (uint64_t)a->batch, BLOCK)) return rc;
    if (int rc = make_map_3d(&p.map_k, a->k, narrow, (uint64_t)a->time, (uint64_t)a->batch, BLOCK)) return rc;
    if (int rc = make_map_3d(&p.map_v, a->v, narrow, (uint64_t)a->time, (uint64_t)a->batch, BLOCK)) return rc;
    if (int rc = make_map_3d(&p.map_do, a->grad_out, wide, (uint64_t)a->time, (uint64_t)a->batch, BLOCK)) return rc;
    p.out_in = (const __nv_bfloat16*)a->out; p.grad_out = (const __nv_bfloat16*)a->grad_out;
    p.lse = (float*)a->lse; p.delta = (float*)a->delta; p.status = device_status_address();
    p.batch = a->batch; p.time = a->time; p.heads = a->heads; p.kv_heads = a->kv_heads;
    const int blocks = (a->time + BLOCK - 1) / BLOCK;
    if (int rc = make_map_3d(&p.map_k2, a->k, narrow, (uint64_t)a->time, (uint64_t)a->batch, DQ_KV)) return rc;
    if (int rc = make_map_3d(&p.map_v2, a->v, narrow, (uint64_t)a->time, (uint64_t)a->batch, DQ_KV)) return rc;
    QMOE_CUDA(cudaFuncSetAttribute(attention_dq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DQ_SMEM));
    QMOE_CUDA(cudaFuncSetAttribute(attention_dkv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DKV_SMEM));
    p.out = (__nv_bfloat16*)a->dq; p.out2 = nullptr;
    chained(attention_dq_kernel, (unsigned)(blocks * a->heads * a->batch), THREADS, DQ_SMEM, stream, p);
    count_tensor_core_launch();
    QMOE_LAUNCH_CHECK("attention_dq_kernel");
    p.out = (__nv_bfloat16*)a->dk; p.out2 = (__nv_bfloat16*)a->dv;
    p.split = dkv_split(a, blocks);
    cudaLaunchConfig_t config = {};
    cudaLaunchAttribute attributes[2] = {chain_attribute()};
    config.gridDim = dim3((unsigned)(blocks * a->kv_heads * a->batch * p.split));
    config.blockDim = dim3(DKV_THREADS);
    config.dynamicSmemBytes = DKV_SMEM;
    config.stream = stream;
    config.attrs = attributes;
    config.numAttrs = p.split > 1 ? 2 : 1;
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim.x = (unsigned)p.split;
    attributes[1].val.clusterDim.y = attributes[1].val.clusterDim.z = 1;
    QMOE_CUDA(cudaLaunchKernelEx(&config, attention_dkv_kernel, p));
    count_tensor_core_launch();
    QMOE_LAUNCH_CHECK("attention_dkv_kernel");
    return 0;
}
