// Shared declarations for libqutai_moe.so (sm_100a only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/qutai_moe.h"

namespace qmoe {

// Rows of every expert group in the permuted ("dispatched") layout are padded to a multiple of
// this, so that a 128-row tensor-core tile never straddles two experts.  Pad rows hold zeros.
constexpr int kRowPad = QMOE_ROW_PAD;
constexpr int kMaxExperts = QMOE_MAX_EXPERTS;
constexpr int kMaxTopK = QMOE_MAX_TOP_K;
// Token rows handled by one block of the routing kernels (8 warps x 4 rows): small blocks keep all SMs
// busy when a rank holds only a few thousand tokens.
constexpr int kRouteRowsPerBlock = 32;

// ---- error plumbing -------------------------------------------------------------------------
void set_error(const char* fmt, ...);
int fail_arg(const char* fmt, ...);                       // returns QMOE_ERR_ARGUMENT
int check_cuda(cudaError_t code, const char* what);       // 0 or positive cudaError_t
#define QMOE_CUDA(expr)                                  \
    do {                                                 \
        int _rc = ::qmoe::check_cuda((expr), #expr);     \
        if (_rc) return _rc;                             \
    } while (0)
#define QMOE_LAUNCH_CHECK(name)                          \
    do {                                                 \
        int _rc = ::qmoe::after_launch(name);            \
        if (_rc) return _rc;                             \
    } while (0)
int after_launch(const char* name);  // cudaGetLastError (+ sync when QUTAI_MOE_SYNC=1) + counters

// per-kernel-class timing (off unless enabled through the ABI)
enum KernelClass {
    KC_ROUTER_GEMM = 0, KC_ROUTE, KC_PERMUTE, KC_EXPERT_GEMM, KC_SWIGLU, KC_COMBINE, KC_COMBINE_BWD,
    KC_WGRAD_GEMM, KC_UNPERMUTE, KC_ROUTE_BWD, KC_CAST, KC_OTHER, KC_EXCHANGE, KC_OPTIMIZER, KC_NORM, KC_ATTENTION,
    KC_HEAD_LOSS, KC_ELEMENTWISE, KC_BARRIER, KC_ALL_REDUCE, KC_COUNT
};
struct TimedScope {  // records a pair of events around the launches made while it is alive
    TimedScope(KernelClass kc, cudaStream_t s);
    ~TimedScope();
    int slot;
    cudaStream_t stream;
};

// ---- kernels in a chain ----------------------------------------------------------------------
// A step is a chain of short kernels on one stream, and between two that follow one another in the ordinary way the device idles
// for about two microseconds: the first drains, its writes are flushed, the second is fetched, its CTAs start and set themselves
// up.  With programmatic dependent launch the second is set up meanwhile and only waits, at chain_wait, until the first has
// completed and its writes are visible.  Every thread of a kernel that is launched through `chained` calls chain_wait before its
// first access to global memory, with one exception below; only its own parameters may be read earlier.  chain_next lets the next kernel of the stream
// start.  It stands behind chain_wait, so at most two kernels are there at a time and whatever lies two launches back is
// complete, and, in a kernel that allocates tensor memory, behind the allocation: the next kernel, if it allocates too, would
// else be able to take the columns first and wait, holding them, for this one.  Without chain_next a kernel lets the next one
// start as its CTAs leave: so do the backward of the combine, the permutation unless a product for few rows follows (permute.cu), and those products unless
// the down product follows for few tokens (gemm_stream.cu).  The CUDA-core products are launched in the ordinary way (see there).
// One kernel reads before its wait: a product for few rows fetches tables (load_l2) and weights (TMA, which reads the L2) that nothing within the
// last launch wrote (gemm_stream.cu).
// 3001 rows, 16 experts, forward and backward (27 launches when this was measured, 21 now): 472 us in ordinary launches, 440 like this; 64 rows over 64
// experts, replayed, L2 flushed: 220 and 215.
// The wait is a volatile statement that clobbers memory, and griddepcontrol.wait is what orders the kernel's loads behind the writes of the
// one before; no load is declared free of order (no __ldg, loads in inline PTX are volatile), and parameters that are const __restrict__ are read
// behind it in program order.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_begin() { chain_wait(); chain_next(); }
// A value that a completed kernel wrote, for a grid that has not waited itself: what a wait makes visible is promised to the grid that waited, and
// an ordinary load may meet a line that the SM kept from an earlier kernel.  The L2 has the write.
__device__ __forceinline__ int load_l2(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
inline cudaLaunchAttribute chain_attribute() {
    cudaLaunchAttribute attribute = {};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    return attribute;
}
// The arguments convert to the kernel's parameters as in an ordinary launch: a pointer of another type does not.  A launch that
// fails is found by the QMOE_LAUNCH_CHECK behind it.
template <typename T> struct AsGiven { using type = T; };
template <typename... Parameters>
inline void chained(void (*kernel)(Parameters...), dim3 grid, dim3 block, size_t shared_bytes, cudaStream_t stream,
                    typename AsGiven<Parameters>::type... arguments) {
    cudaLaunchAttribute attribute = chain_attribute();
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = shared_bytes;
    config.stream = stream;
    config.attrs = &attribute;
    config.numAttrs = 1;
    (void)cudaLaunchKernelEx(&config, kernel, arguments...);
}

// ---- small device helpers -------------------------------------------------------------------
template <typename T> struct Act;
template <> struct Act<float> {
    static __device__ __forceinline__ float load(const float* p) { return *p; }
    static __device__ __forceinline__ void store(float* p, float v) { *p = v; }
    static constexpr int kVec = 4;  // elements per 16-byte access
};
template <> struct Act<__nv_bfloat16> {
    static __device__ __forceinline__ float load(const __nv_bfloat16* p) { return __bfloat162float(*p); }
    static __device__ __forceinline__ void store(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
    static constexpr int kVec = 8;
};

// 16-byte vector of activations unpacked to floats and back
template <typename T> struct Vec16;
template <> struct Vec16<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void unpack(const uint4& v, float* f) {
        f[0] = __uint_as_float(v.x); f[1] = __uint_as_float(v.y);
        f[2] = __uint_as_float(v.z); f[3] = __uint_as_float(v.w);
    }
    static __device__ __forceinline__ uint4 pack(const float* f) {
        return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
    }
};
template <> struct Vec16<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void unpack(const uint4& v, float* f) {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[2 * i] = __uint_as_float(w[i] << 16);
            f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
    static __device__ __forceinline__ uint4 pack(const float* f) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
            w[i] = *reinterpret_cast<uint32_t*>(&h);
        }
        return make_uint4(w[0], w[1], w[2], w[3]);
    }
};

__device__ __forceinline__ float sigmoid_stable(float v) {
    // two-branch logistic: never exponentiates a positive number
    if (v >= 0.f) return 1.f / (1.f + __expf(-v));
    float e = __expf(v);
    return e / (1.f + e);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Warps that share a token row in the row kernels (permute, combine): one where the tokens alone fill the machine, up to 8
// (each with at least one 16-byte piece per lane) for a handful of tokens, where a row's serial chain of loads is the
// kernel's time (64 rows of 2048: permute 9.2 -> 4 us, combine 9.0 -> 4 us).
inline int part_bits_per_row(long long tokens, long long pieces) {      // log2 of the warps per row
    int bits = 0;
    while (bits < 3 && (tokens << bits) < 2048 && pieces > (32ll << bits)) ++bits;
    return bits;
}

// Zero rows count .. round_up(count, 2^pad_bits) - 1 of every expert's group (2^pad_bits divides kRowPad), a warp per row.
// Shifts throughout, here and for the warps of a row: a 64-bit division per row cost 64 tokens over 256 experts a tenth of the
// permute (12.3 -> 14.3 us).
template <typename T, bool VEC>
__device__ __forceinline__ void zero_pad_rows(T* out, const int* offsets, const int* counts, int experts, int pad_bits, long long width,
                                              int warp, int nwarps) {
    const int lane = threadIdx.x & 31, pad = 1 << pad_bits;
    for (int i = warp; i < experts << pad_bits; i += nwarps) {
        const int e = i >> pad_bits, count = counts[e], row = count + (i & (pad - 1));
        if (row >= (count + pad - 1 & -pad)) continue;
        T* dst = out + ((long long)offsets[e] + row) * width;
        if constexpr (VEC) {
            constexpr int N = Vec16<T>::N;
            for (int c = lane; c < (int)(width / N); c += 32) *reinterpret_cast<uint4*>(dst + (long long)c * N) = make_uint4(0, 0, 0, 0);
        } else {
            for (long long c = lane; c < width; c += 32) Act<T>::store(dst + c, 0.f);
        }
    }
}

// this warp's sum of squares of a row of 16-byte pieces, in every lane: the order is part of the norm's result
template <typename T> __device__ __forceinline__ float row_square_sum(const T* src, long long width) {
    constexpr int N = Vec16<T>::N;
    float total = 0.f;
    for (int c = threadIdx.x & 31; c < (int)(width / N); c += 32) {
        float f[N];
        Vec16<T>::unpack(*reinterpret_cast<const uint4*>(src + (long long)c * N), f);
#pragma unroll
        for (int i = 0; i < N; ++i) total = fmaf(f[i], f[i], total);
    }
    return warp_sum(total);
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
}
// One router logit by one warp, in every lane: row . w, with the lanes striding over the width and a fixed shuffle tree.  Four 16-byte loads of
// the weight row and of the token row are in flight per lane and iteration, so the few round trips to L2 overlap.
// NORM: the logit of the normalised row, inv * (row . (w * norm weight)), with inv = 1 / rms from the same pass over the row.
template <typename T, bool NORM>
__device__ __forceinline__ float small_logit(const T* row, const float* we, long long d, const float* norm_weight, float eps, float& inv) {
    const int lane = threadIdx.x & 31;
    const bool vec = (d & 3) == 0 && (((uintptr_t)row | (uintptr_t)we | (NORM ? (uintptr_t)norm_weight : 0)) & 15u) == 0;
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f, square = 0.f;
    if (vec) {
        for (long long j = (long long)lane * 4; j < d; j += 512) {
            float4 wv[4], xv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const long long at = j + 128 * u;
                const bool in = at < d;
                wv[u] = in ? load4(we + at) : make_float4(0.f, 0.f, 0.f, 0.f);
                xv[u] = in ? load4(row + at) : make_float4(0.f, 0.f, 0.f, 0.f);
                if (NORM && in) {
                    const float4 nv = load4(norm_weight + at);
                    wv[u].x *= nv.x; wv[u].y *= nv.y; wv[u].z *= nv.z; wv[u].w *= nv.w;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {   // fixed order: the sums do not depend on timing
                a0 = fmaf(xv[u].x, wv[u].x, a0);
                a1 = fmaf(xv[u].y, wv[u].y, a1);
                a2 = fmaf(xv[u].z, wv[u].z, a2);
                a3 = fmaf(xv[u].w, wv[u].w, a3);
                if (NORM) square = fmaf(xv[u].w, xv[u].w, fmaf(xv[u].z, xv[u].z, fmaf(xv[u].y, xv[u].y, fmaf(xv[u].x, xv[u].x, square))));
            }
        }
    } else {
        for (long long j = lane; j < d; j += 32) {
            const float v = Act<T>::load(row + j);
            a0 = fmaf(v, NORM ? we[j] * norm_weight[j] : we[j], a0);
            if (NORM) square = fmaf(v, v, square);
        }
    }
    float acc = (a0 + a1) + (a2 + a3);
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, step);
    if (NORM) {
        inv = rsqrtf(warp_sum(square) / (float)d + eps);
        acc *= inv;
    }
    return acc;
}

inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }
int sm_count();

// ---- CUDA-core GEMM descriptor (gemm_simt.cu) ------------------------------------------------
enum SimtGroupMode { SG_PLAIN = 0, SG_ROWS = 1, SG_K = 2, SG_SPLITK = 3 };
struct SimtGemmArgs {
    const void* A;
    const void* B;
    void* C;
    const void* A2;  // optional second segment (same shapes and strides), may be null
    const void* B2;
    long long M, N, K;
    long long a_rs, a_cs;  // A(m, k) = A[m * a_rs + k * a_cs]
    long long b_rs, b_cs;  // B(k, n) = B[k * b_rs + n * b_cs]
    long long ldc;         // C(m, n) = C[m * ldc + n]
    int accumulate;
    int mode;
    const int* tile_expert;  // SG_ROWS: expert of each kRowPad-row tile of the dispatched layout
    const int* offsets;      // SG_K: first dispatched row of each expert
    const int* counts;       // SG_K: rows of each expert
    const int* meta;         // SG_ROWS: meta[0] = dispatched rows in use
    long long b_slab;        // SG_ROWS: elements of B per expert
    long long c_slab;        // SG_K / SG_SPLITK: elements of C per expert / per split
    long long k_chunk;       // SG_SPLITK: K handled by one split
    long long row_tiles[3];  // SG_ROWS: 128-row tiles in use, guesses for the choice of a kernel (0: ceil(M / 128))
    long long mean_rows;     // SG_K: rows of an expert, on average
};
// dtype codes QMOE_F32 / QMOE_BF16 for A, B, C; m_extent = rows the grid must cover
int launch_simt_gemm(const SimtGemmArgs& g, int a_dtype, int b_dtype, int c_dtype, long long m_extent, int groups,
                     cudaStream_t stream);
// up to kSimtProducts products of one mode, one set of groups and the same operand types (m_extent: g.M), in one launch where they take the tiles
constexpr int kSimtProducts = 3;
int launch_simt_gemms(const SimtGemmArgs* g, int count, int a_dtype, int b_dtype, int c_dtype, int groups, cudaStream_t stream);

// ---- cross-file entry points -----------------------------------------------------------------
// qmoe_permute / qmoe_permute_norm with the pad rows zeroed only up to a multiple of `pad` rows per expert; let_next: the next kernel may start early
int launch_permute(const qmoe_route_t* r, uint64_t x, uint64_t out, int32_t dtype, int64_t width, int pad, bool let_next, uint64_t stream);
int launch_permute_norm(const qmoe_route_t* r, uint64_t x, uint64_t inverse, uint64_t weight, uint64_t out, int32_t dtype, int64_t width, int pad,
                        uint64_t stream);
// router_forward (with norm_weight router_forward_norm) and the routing in one launch, for a handful of logits (router_route_ok)
bool router_route_ok(const qmoe_route_t* r);
int router_route_small(const qmoe_route_t* r, uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t norm_weight, double eps, uint64_t inverse, uint64_t scores,
                       int64_t width, uint64_t stream);
bool router_norm_ok(int64_t tokens, int32_t experts, int64_t width, int32_t x_dtype, uint64_t x, uint64_t scratch);
int router_forward_norm(uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t norm_weight, double eps, uint64_t inverse, uint64_t scores,
                        int64_t tokens, int64_t width, int32_t experts, uint64_t stream);
// the same on the tensor cores, for any number of tokens (router_tensor_cores): the logits of the normalised rows from the raw ones
bool router_tensor_cores(int32_t x_dtype, int32_t experts, int64_t width, uint64_t x, uint64_t scratch);
int router_forward_scaled(uint64_t x, uint64_t w_router, uint64_t norm_weight, double eps, uint64_t inverse, uint64_t scores, uint64_t scratch,
                          int64_t tokens, int64_t width, int32_t experts, uint64_t stream);
int router_backward_scaled(uint64_t d_scores, uint64_t row_scale, uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t dx_router,
                           uint64_t d_w_router, uint64_t col_scale, uint64_t scratch, int64_t tokens, int64_t width, int32_t experts, uint64_t stream);
int route_check(const qmoe_route_t* r);
int launch_swiglu(const qmoe_route_t* r, uint64_t g, uint64_t u, uint64_t h, int dtype, long long hidden, cudaStream_t stream);
int launch_swiglu_backward(const qmoe_route_t* r, uint64_t dh, uint64_t g, uint64_t u, uint64_t dg, uint64_t du, int dtype,
                           long long hidden, cudaStream_t stream);
bool tcgen05_shape_ok(long long width, long long hidden);
int tc_swiglu_forward(const qmoe_route_t* r, const qmoe_experts_t* ex, uint64_t x, uint64_t g, uint64_t u, uint64_t h, cudaStream_t stream);
// optional "store each output row at its return address on the rank that owns it" for the bf16 row products
struct TcScatter {
    const int* ret;                 // [rows] rank << 26 | row
    unsigned long long base[16];    // destination buffer of every rank
};
int tc_rows_nt(const qmoe_route_t* r, int experts, uint64_t a, uint64_t b, uint64_t c, long long K, long long N, cudaStream_t stream,
               const TcScatter* scatter = nullptr, long long rows = 0);
int tc_rows_nn(const qmoe_route_t* r, int experts, uint64_t a, uint64_t b, uint64_t a2, uint64_t b2, uint64_t c, long long K,
               long long N, cudaStream_t stream, const TcScatter* scatter = nullptr, long long rows = 0);
// the same two forward products for few rows per expert (gemm_stream.cu)
// pad_rows: every pad row holds zeros afterwards; else (QMOE_EXPERTS_SHORT_PADS) only those up to a multiple of kStreamPad rows of each expert
// early: the kernel before on the stream is this call's own and wrote neither the tables nor the weights (see the kernel)
constexpr int kStreamPad = 16;
bool stream_shape_ok(const qmoe_route_t* r, const qmoe_experts_t* ex);
bool stream_down_early(const qmoe_route_t* r, const qmoe_experts_t* ex);     // the down product starts beside the up product's tail
int stream_swiglu_forward(const qmoe_route_t* r, const qmoe_experts_t* ex, uint64_t x, uint64_t g, uint64_t u, uint64_t h, bool pad_rows, bool early, bool let_next,
                          cudaStream_t stream);
int stream_rows_nt(const qmoe_route_t* r, int experts, uint64_t a, uint64_t b, uint64_t c, long long K, long long N, bool pad_rows, bool early,
                   cudaStream_t stream);
int tc_dswiglu(const qmoe_route_t* r, int experts, uint64_t dy, uint64_t w_down, uint64_t g, uint64_t u, uint64_t dg,
               uint64_t du, long long d, long long h, cudaStream_t stream);
int tc_wgrad3(const qmoe_route_t* r, int experts, uint64_t dy, uint64_t h_act, uint64_t x, uint64_t dg, uint64_t du,
              uint64_t d_w_down, uint64_t d_w_gate, uint64_t d_w_up, long long d, long long h, cudaStream_t stream);
int tc_wgrad1(const qmoe_route_t* r, uint64_t a, uint64_t b, uint64_t out, long long M, long long N, cudaStream_t stream,
              int groups = 1, long long slab = 0, int sum_rows = 0);
int tc_router_forward(uint64_t x, uint64_t w3, uint64_t scores, uint64_t row_scale, long long T, long long d, int E, int S, cudaStream_t stream);
int tc_plain_f32_nn(uint64_t a, uint64_t b, uint64_t c, long long T, long long K, long long N, cudaStream_t stream);
int tc_split_wgrad(uint64_t a, long long a_pitch, uint64_t b, uint64_t partial, const int* offsets, const int* counts,
                   int splits, long long T, long long M, long long N, cudaStream_t stream);
int simt_router_logits(uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t scores, int64_t tokens, int64_t width,
                       int32_t experts, cudaStream_t stream);
int simt_router_backward(uint64_t d_scores, uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t dx_router,
                         uint64_t d_w_router, uint64_t partials, int64_t tokens, int64_t width, int32_t experts,
                         cudaStream_t stream);
long long simt_router_partials(int64_t tokens, int32_t experts, int64_t width);
int launch_reduce_partials(const float* partials, float* out, long long n, int splits, cudaStream_t stream);
void count_tensor_core_launch();
int kernel_variant(int which);  // 0 = default form, 1 = the comparison form selected by qmoe_test_select_variant
int* device_status_address();

}  // namespace qmoe
