// Router projection (scores = x W_r^T) and its backward, in fp32 semantics.
//
// Upstream runs the router under `set_matmul_precision(None)` (src/qutai/lm/layers.py:377-378): fp32
// weights, fp32 arithmetic, whatever the activation dtype.  Two implementations sit behind the same
// entry points:
//   * bf16 activations: the tensor cores, with every fp32 factor split into bf16 terms
//     (v = hi + mid + lo, 8 mantissa bits each, so hi + mid + lo carries all 24).  bf16 x bf16
//     products are exact in fp32 and the accumulation is fp32, so the result differs from an fp32
//     FMA chain only by fp32 rounding of the partial sums.  x itself is bf16 and needs no split.
//       scores      = x . (W_hi + W_mid + W_lo)^T                       one launch, K = d
//       dx_router   = ds . W_hi + (ds_hi + ds_mid) . W_mid              one launch, K = 6 S
//       dW_router   = (ds_hi + ds_mid + ds_lo)^T . x                    split over token blocks, reduced in a fixed order
//   * fp32 activations (or more than 64 experts): the CUDA-core GEMM of gemm_simt.cu.
#include "common.cuh"

namespace qmoe {
namespace {

constexpr long long kAlign = 256;
inline long long align_up(long long v) { return (v + kAlign - 1) / kAlign * kAlign; }

struct RouterScratch {  // byte offsets inside the caller's scratch buffer
    int S, splits;
    long long rows_per_split;
    long long w3, wbwd, ds6, tables, partial, total;
};

RouterScratch plan_scratch(long long T, int E, long long d) {
    RouterScratch r;
    r.S = (E + 31) / 32 * 32;
    // Ranges of the tokens for the weight gradient: its [3 S, d] product is a few tiles of 128 x 256, so the ranges are what
    // spreads it over the SMs, against the sum over them afterwards (16 experts, d 1024, product + sum: 3001 tokens 19 us in 2
    // ranges, 15 in 11; 16384 tokens 25 us in 16, 27 in 32).
    long long splits = T / 256 < 16 ? T / 256 : 16;
    if (splits < T / 1024) splits = T / 1024;
    if (splits < 1) splits = 1;
    if (splits > 32) splits = 32;
    const long long room = splits;     // sizes that never shrink as T grows: rounded to whole tiles, fewer ranges may be enough (3840
                                       // tokens 15, 4095 tokens 11), and a scratch made for the most tokens serves fewer
    r.rows_per_split = ((T + splits - 1) / splits + kRowPad - 1) / kRowPad * kRowPad;
    r.splits = (int)((T + r.rows_per_split - 1) / r.rows_per_split);
    long long at = 0;
    r.w3 = at;      at = align_up(at + 3ll * r.S * d * 2);
    r.wbwd = at;    at = align_up(at + 6ll * r.S * d * 2);
    r.ds6 = at;     at = align_up(at + T * 6ll * r.S * 2);
    r.tables = at;  at = align_up(at + (2ll * room + 1) * 4);
    r.partial = at; at = align_up(at + room * 3 * r.S * d * 4);
    r.total = at;
    return r;
}

bool tc_router_ok(int x_dtype, int E, long long d, uint64_t x, uint64_t scratch) {
    return x_dtype == QMOE_BF16 && E <= 64 && d % 8 == 0 && d >= 64 && scratch && !(x & 15u) && !(scratch & 255u);
}

__device__ __forceinline__ void split3(float v, __nv_bfloat16& hi, __nv_bfloat16& mid, __nv_bfloat16& lo) {
    hi = __float2bfloat16_rn(v);
    const float r1 = v - __bfloat162float(hi);
    mid = __float2bfloat16_rn(r1);
    lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
}

// Elements first, first + step, ... of W [E, d] fp32 (times col_scale[j], when given) -> w3 [3S, d] = {hi; mid; lo} (forward), or wbwd [6S, d] = {hi; hi; hi; mid; mid; 0}
// (backward); rows E..S-1 zero
__device__ __forceinline__ void split_w(const float* __restrict__ w, const float* __restrict__ col_scale, __nv_bfloat16* __restrict__ w3,
                                        __nv_bfloat16* __restrict__ wbwd, int E, int S, long long d, long long first, long long step) {
    const long long n = (long long)S * d;
    const __nv_bfloat16 zero = __float2bfloat16_rn(0.f);
    for (long long i = first; i < n; i += step) {
        const long long r = i / d;
        __nv_bfloat16 hi, mid, lo;
        float v = r < E ? w[i] : 0.f;
        if (col_scale && r < E) v *= col_scale[i - r * d];
        split3(v, hi, mid, lo);
        if (w3) { w3[i] = hi; w3[n + i] = mid; w3[2 * n + i] = lo; }
        if (wbwd) { wbwd[i] = hi; wbwd[n + i] = hi; wbwd[2 * n + i] = hi; wbwd[3 * n + i] = mid; wbwd[4 * n + i] = mid; wbwd[5 * n + i] = zero; }
    }
}

// What the forward's product needs: the weight terms, by the first w_blocks blocks, and with x the inverse of every row's norm, by a warp per
// row of the others.  One launch each and one for the weight times the norm weight were three, and the scaled logits a fourth behind the
// product: block of 3001 rows, 16 experts, 1024 x 2048, forward and backward 429 -> 427 us, with the backward's two below in one.
__global__ void __launch_bounds__(256)
router_prepare_kernel(const float* __restrict__ w, const float* __restrict__ col_scale, __nv_bfloat16* __restrict__ w3, int E, int S, long long d, int w_blocks,
                      const __nv_bfloat16* __restrict__ x, float* __restrict__ inverse, long long tokens, float eps) {
    chain_begin();
    if ((int)blockIdx.x < w_blocks) {
        split_w(w, col_scale, w3, nullptr, E, S, d, (long long)blockIdx.x * blockDim.x + threadIdx.x, (long long)w_blocks * blockDim.x);
        return;
    }
    const long long warp = (long long)(blockIdx.x - w_blocks) * 8 + (threadIdx.x >> 5), warps = (long long)(gridDim.x - w_blocks) * 8;
    for (long long t = warp; t < tokens; t += warps) {
        const float total = row_square_sum(x + t * d, d);
        if ((threadIdx.x & 31) == 0) inverse[t] = rsqrtf(total / (float)d + eps);
    }
}

// What the backward's products need: the weight terms, by the first w_blocks blocks; by the others ds [T, E] fp32 (first multiplied by
// row_scale[t] in place, when given) -> ds6 [T, 6S] = {hi | mid | lo | hi | mid | 0}; also the token-block tables of the split contraction
__global__ void __launch_bounds__(256)
router_split_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ wbwd, long long d, int w_blocks, float* __restrict__ ds,
                    const float* __restrict__ row_scale, __nv_bfloat16* __restrict__ ds6, long long T, int E, int S,
                    int* __restrict__ tables, int splits, long long rows_per_split) {
    chain_begin();
    if (blockIdx.x == 0 && threadIdx.x <= splits) {
        const int i = threadIdx.x;
        tables[i] = (int)(i * rows_per_split);  // offsets[splits + 1]
        if (i < splits) {
            long long c = T - i * rows_per_split;
            tables[splits + 1 + i] = (int)(c < 0 ? 0 : (c > rows_per_split ? rows_per_split : c));  // counts[splits]
        }
    }
    if ((int)blockIdx.x < w_blocks) {
        split_w(w, nullptr, nullptr, wbwd, E, S, d, (long long)blockIdx.x * blockDim.x + threadIdx.x, (long long)w_blocks * blockDim.x);
        return;
    }
    const long long n = T * S;
    const __nv_bfloat16 zero = __float2bfloat16_rn(0.f);
    for (long long i = (long long)(blockIdx.x - w_blocks) * blockDim.x + threadIdx.x; i < n; i += (long long)(gridDim.x - w_blocks) * blockDim.x) {
        const long long t = i / S;
        const int e = (int)(i - t * S);
        __nv_bfloat16 hi, mid, lo;
        float value = e < E ? ds[t * E + e] : 0.f;
        if (row_scale && e < E) {
            value *= row_scale[t];
            ds[t * E + e] = value;      // no other thread has this element
        }
        split3(value, hi, mid, lo);
        __nv_bfloat16* row = ds6 + t * 6 * S;
        row[e] = hi; row[S + e] = mid; row[2 * S + e] = lo; row[3 * S + e] = hi; row[4 * S + e] = mid; row[5 * S + e] = zero;
    }
}

// dW [E, d] = sum over splits and over the three term groups, in a fixed order (times col_scale[j], when given)
__global__ void __launch_bounds__(256)
router_reduce_dw_kernel(const float* __restrict__ partial, const float* __restrict__ col_scale, float* __restrict__ dw, int E, int S, long long d,
                        int splits) {
    chain_begin();
    const long long n = (long long)E * d;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long e = i / d, j = i - e * d;
        float acc = 0.f;
        for (int s = 0; s < splits; ++s) {
            const float* slab = partial + (long long)s * 3 * S * d;
            acc += (slab[(2 * S + e) * d + j] + slab[(S + e) * d + j]) + slab[e * d + j];
        }
        dw[i] = col_scale ? acc * col_scale[j] : acc;
    }
}

// Few tokens (decode): one block per token, a warp per expert in turn, fp32 dot products with the lanes
// striding over the width and a fixed shuffle tree, so the logits are run-to-run identical.  A tile kernel
// would put the whole product on one or two SMs and walk the width serially.
// The warps of a token read every weight row again, from L2: up to 512 tokens that is the shorter way whatever the sizes (a call of 600
// tokens, 32 experts, d 584, with the norm: 40 us, 43 with the logits on the tensor cores).  Beyond them by an estimate of both ways, in us beyond
// what a launch takes, fitted to 600 .. 65536 tokens, 1 .. 128 experts, widths 64 .. 4096 with L2 flushed: this kernel takes a
// block's issue per 8 logits (16384 x 16 x 64: 46 us) or the weight reads (32768 x 16 x 2048: 293); three times that when the
// width is no multiple of 4, half as much again with the norm; the tile kernel a chain of `width` products per tile until its
// tiles fill the machine (16 and 212); the tensor cores two launches and little else (bf16, 16384 x 16 x 64: 13, against 50 here).
// With the norm the CUDA cores' other way has three launches more, 9 us.  The tensor cores' has none more (router_forward_scaled) and by time would
// be worth 3: of what the 9 leave here, calls of 1000 x 64 x 256 take 45 us and 41 there, 2000 x 32 x 256 51 and 44, 4000 x 16 x 256 52 and 44, 8000 x 8 x 256 56 and 47.  They stay
// for their precision: the logits' error here is 0.97e-7 of their norm, there 2.3e-7 (width 256; 4.7e-7 at 512).
constexpr long long kSmallRouterTokens = 512, kSmallRouterProducts = 1ll << 24;
bool small_router(long long tokens, int experts, long long width, int x_dtype, bool tensor_cores, bool norm) {
    if (tokens <= kSmallRouterTokens) return true;
    if (tokens * experts * width > kSmallRouterProducts && !(x_dtype == QMOE_F32 && experts <= 16)) return false;
    const double T = (double)tokens, d = (double)width;
    const double blocks = T * (4.5e-4 * ((experts + 7) / 8) + 1e-4 * experts), reads = T * experts * (3e-5 + 2.7e-7 * d);
    const double here = (blocks > reads ? blocks : reads) * (width % 4 ? 3 : 1) * (norm ? 1.5 : 1);
    const double there = tensor_cores ? 6 + 5.6e-3 * d + 6e-7 * T * d : 7.5e-2 * d * (T > 30000 ? T / 30000 : 1);
    return here <= there + (norm ? 9 : 0);
}
// grid (tokens, ceil(E / 8)): warp w of block (t, g) computes scores[t, 8 g + w]
template <typename T, bool NORM>
__global__ void __launch_bounds__(256)
router_small_kernel(const T* __restrict__ x, const float* __restrict__ w, float* __restrict__ scores, int E, long long d,
                    const float* __restrict__ norm_weight, float eps, float* __restrict__ inverse) {
    chain_begin();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = blockIdx.y * 8 + warp;
    if (e >= E) return;
    float inv = 0.f;
    const float acc = small_logit<T, NORM>(x + (long long)blockIdx.x * d, w + (long long)e * d, d, norm_weight, eps, inv);
    if (NORM && lane == 0 && e == 0) inverse[blockIdx.x] = inv;
    if (lane == 0) scores[(long long)blockIdx.x * E + e] = acc;
}

int elem_grid(long long n) {
    long long blocks = (n + 255) / 256;
    const long long cap = (long long)sm_count() * 8;
    return (int)(blocks > cap ? cap : (blocks < 1 ? 1 : blocks));
}

}  // namespace
}  // namespace qmoe

using namespace qmoe;

extern "C" int64_t qmoe_router_scratch_bytes(int64_t tokens, int32_t experts, int64_t width) {
    if (tokens <= 0 || experts <= 0 || width <= 0) return 0;
    const long long simt = simt_router_partials(tokens, experts, width) * 4;
    const long long tc = plan_scratch(tokens, experts, width).total;
    return simt > tc ? simt : tc;
}

extern "C" int64_t qmoe_router_grad_partials(int64_t tokens, int32_t experts, int64_t width) {
    return (qmoe_router_scratch_bytes(tokens, experts, width) + 3) / 4;
}

extern "C" int qmoe_router_forward(uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t scores, uint64_t scratch,
                                   int64_t tokens, int64_t width, int32_t experts, uint64_t stream_) {
    if (!x || !w_router || !scores) return fail_arg("router_forward: null address");
    if (tokens <= 0 || width <= 0 || experts <= 0) return fail_arg("router_forward: sizes must be positive");
    if (x_dtype != QMOE_F32 && x_dtype != QMOE_BF16) return fail_arg("router_forward: bad dtype %d", x_dtype);
    cudaStream_t stream = (cudaStream_t)stream_;
    const bool tensor_cores = tc_router_ok(x_dtype, experts, width, x, scratch);
    if (small_router(tokens, experts, width, x_dtype, tensor_cores, false)) {
        TimedScope timed(KC_ROUTER_GEMM, stream);
        const dim3 grid((unsigned)tokens, (unsigned)((experts + 7) / 8));
        if (x_dtype == QMOE_BF16)
            chained(router_small_kernel<__nv_bfloat16, false>, grid, 256, 0, stream, (const __nv_bfloat16*)x, (const float*)w_router, (float*)scores,
                                                                                experts, width, nullptr, 0.f, nullptr);
        else
            chained(router_small_kernel<float, false>, grid, 256, 0, stream, (const float*)x, (const float*)w_router, (float*)scores, experts, width,
                                                                        nullptr, 0.f, nullptr);
        QMOE_LAUNCH_CHECK("router_small_kernel");
        return 0;
    }
    if (!tensor_cores)
        return simt_router_logits(x, x_dtype, w_router, scores, tokens, width, experts, stream);
    TimedScope timed(KC_ROUTER_GEMM, stream);
    const RouterScratch r = plan_scratch(tokens, experts, width);
    const int w_blocks = elem_grid((long long)r.S * width);
    chained(router_prepare_kernel, w_blocks, 256, 0, stream, (const float*)w_router, nullptr, (__nv_bfloat16*)(scratch + r.w3), experts, r.S, width, w_blocks,
            nullptr, nullptr, 0, 0.f);
    QMOE_LAUNCH_CHECK("router_prepare_kernel");
    return tc_router_forward(x, scratch + r.w3, scores, 0, tokens, width, experts, r.S, stream);
}

bool qmoe::router_tensor_cores(int32_t x_dtype, int32_t experts, int64_t width, uint64_t x, uint64_t scratch) {
    return tc_router_ok(x_dtype, experts, width, x, scratch);
}

int qmoe::router_forward_scaled(uint64_t x, uint64_t w_router, uint64_t norm_weight, double eps, uint64_t inverse, uint64_t scores, uint64_t scratch,
                                int64_t tokens, int64_t width, int32_t experts, uint64_t stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_ROUTER_GEMM, stream);
    const RouterScratch r = plan_scratch(tokens, experts, width);
    const int w_blocks = elem_grid((long long)r.S * width), row_blocks = elem_grid(tokens * 32);
    chained(router_prepare_kernel, w_blocks + row_blocks, 256, 0, stream, (const float*)w_router, (const float*)norm_weight, (__nv_bfloat16*)(scratch + r.w3),
            experts, r.S, width, w_blocks, (const __nv_bfloat16*)x, (float*)inverse, tokens, (float)eps);
    QMOE_LAUNCH_CHECK("router_prepare_kernel");
    return tc_router_forward(x, scratch + r.w3, scores, inverse, tokens, width, experts, r.S, stream);
}

bool qmoe::router_norm_ok(int64_t tokens, int32_t experts, int64_t width, int32_t x_dtype, uint64_t x, uint64_t scratch) {
    return small_router(tokens, experts, width, x_dtype, tc_router_ok(x_dtype, experts, width, x, scratch), true);
}

// inverse[t] and the logits of the normalised rows in one launch (tokens within router_norm_ok)
int qmoe::router_forward_norm(uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t norm_weight, double eps, uint64_t inverse, uint64_t scores,
                              int64_t tokens, int64_t width, int32_t experts, uint64_t stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_ROUTER_GEMM, stream);
    const dim3 grid((unsigned)tokens, (unsigned)((experts + 7) / 8));
    if (x_dtype == QMOE_BF16)
        chained(router_small_kernel<__nv_bfloat16, true>, grid, 256, 0, stream, (const __nv_bfloat16*)x, (const float*)w_router, (float*)scores, experts, width,
                                                                           (const float*)norm_weight, (float)eps, (float*)inverse);
    else
        chained(router_small_kernel<float, true>, grid, 256, 0, stream, (const float*)x, (const float*)w_router, (float*)scores, experts, width,
                                                                   (const float*)norm_weight, (float)eps, (float*)inverse);
    QMOE_LAUNCH_CHECK("router_small_kernel");
    return 0;
}

extern "C" int qmoe_router_logits(uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t scores, int64_t tokens,
                                  int64_t width, int32_t experts, uint64_t stream) {
    return qmoe_router_forward(x, x_dtype, w_router, scores, 0, tokens, width, experts, stream);
}

extern "C" int qmoe_router_backward(uint64_t d_scores, uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t dx_router,
                                    uint64_t d_w_router, uint64_t scratch, int64_t tokens, int64_t width, int32_t experts,
                                    uint64_t stream) {
    return router_backward_scaled(d_scores, 0, x, x_dtype, w_router, dx_router, d_w_router, 0, scratch, tokens, width, experts, stream);
}

// The same for d_scores[t, :] * row_scale[t], which d_scores holds afterwards, with the weight gradient's columns multiplied by
// col_scale (0: neither).  The scales ride along where the factors are split and the ranges are summed.
int qmoe::router_backward_scaled(uint64_t d_scores, uint64_t row_scale, uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t dx_router,
                                 uint64_t d_w_router, uint64_t col_scale, uint64_t scratch, int64_t tokens, int64_t width, int32_t experts,
                                 uint64_t stream_) {
    if (!d_scores || !x || !w_router) return fail_arg("router_backward: null address");
    if (tokens <= 0 || width <= 0 || experts <= 0) return fail_arg("router_backward: sizes must be positive");
    if (x_dtype != QMOE_F32 && x_dtype != QMOE_BF16) return fail_arg("router_backward: bad dtype %d", x_dtype);
    cudaStream_t stream = (cudaStream_t)stream_;
    if (!tc_router_ok(x_dtype, experts, width, x, scratch)) {
        if (row_scale)
            if (int rc = qmoe_scale_f32(d_scores, d_scores, row_scale, 0, tokens, experts, stream_)) return rc;
        if (int rc = simt_router_backward(d_scores, x, x_dtype, w_router, dx_router, d_w_router, scratch, tokens, width, experts, stream)) return rc;
        return col_scale && d_w_router ? qmoe_scale_f32(d_w_router, d_w_router, 0, col_scale, experts, width, stream_) : 0;
    }
    TimedScope timed(KC_ROUTER_GEMM, stream);
    const RouterScratch r = plan_scratch(tokens, experts, width);
    const int S = r.S;
    int* tables = (int*)(scratch + r.tables);
    const int w_blocks = elem_grid((long long)S * width);
    chained(router_split_kernel, w_blocks + elem_grid(tokens * S), 256, 0, stream, (const float*)w_router, (__nv_bfloat16*)(scratch + r.wbwd), width, w_blocks,
            (float*)d_scores, (const float*)row_scale, (__nv_bfloat16*)(scratch + r.ds6), tokens, experts, S, tables, r.splits, r.rows_per_split);
    QMOE_LAUNCH_CHECK("router_split_kernel");
    if (dx_router)
        if (int rc = tc_plain_f32_nn(scratch + r.ds6, scratch + r.wbwd, dx_router, tokens, 6ll * S, width, stream)) return rc;
    if (d_w_router) {
        if (int rc = tc_split_wgrad(scratch + r.ds6, 6ll * S, x, scratch + r.partial, tables, tables + r.splits + 1, r.splits,
                                    tokens, 3ll * S, width, stream)) return rc;
        chained(router_reduce_dw_kernel, elem_grid((long long)experts * width), 256, 0, stream, 
            (const float*)(scratch + r.partial), (const float*)col_scale, (float*)d_w_router, experts, S, width, r.splits);
        QMOE_LAUNCH_CHECK("router_reduce_dw_kernel");
    }
    return 0;
}
