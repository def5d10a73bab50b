// The small memory-bound operations around attention and the feed-forward half of a decoder block, with upstream's
// meaning of every argument (src/qutai/backends/cuda_lm.py, kernels src/qutai/backends/cuda/lm.cu:11-64, CPU statements
// src/qutai/backends/cpu_lm.py:54-140): RMS norm and its backward, rotary position embedding, the token embedding and
// its backward.  Upstream launches one 256-thread block per row (norm) or one thread per element with scalar accesses;
// here a warp owns a row and moves 16 or 32 bytes per lane per access in the norm, the norm weight's gradient is reduced in a fixed
// order (no floating-point atomics), and the embedding's backward walks each token's positions in order, as
// upstream's does, so every result is the same on every run.
#include <stdlib.h>

#include <type_traits>

#include "common.cuh"

namespace qmoe {
namespace {

constexpr int kThreads = 256;
constexpr int kWarpsPerBlock = kThreads / 32;
constexpr int kSlabRows = 32;          // rows of one block of the norm weight's gradient

int row_grid(long long rows) {
    const long long blocks = (rows + kWarpsPerBlock - 1) / kWarpsPerBlock;
    return (int)(blocks > 8ll * 148 ? 8 * 148 : (blocks < 1 ? 1 : blocks));
}
int flat_grid(long long n) {
    const long long blocks = (n + kThreads - 1) / kThreads;
    return (int)(blocks > 8ll * 148 ? 8 * 148 : (blocks < 1 ? 1 : blocks));
}

// eight consecutive elements per lane and access: 16 bytes of bf16, 32 bytes of fp32
__device__ __forceinline__ void load8(const float* p, float* f) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float* f) { Vec16<__nv_bfloat16>::unpack(*reinterpret_cast<const uint4*>(p), f); }
__device__ __forceinline__ void store8(float* p, const float* f) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(f[4], f[5], f[6], f[7]);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float* f) { *reinterpret_cast<uint4*>(p) = Vec16<__nv_bfloat16>::pack(f); }

// eight elements as they lie in memory, converted when they are used (keeps many loads in flight in few registers)
template <typename T> struct Raw8;
template <> struct Raw8<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float* p) { a = *reinterpret_cast<const float4*>(p); b = *reinterpret_cast<const float4*>(p + 4); }
    __device__ __forceinline__ void unpack(float* f) const { f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w; }
};
template <> struct Raw8<__nv_bfloat16> {
    uint4 v;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ void unpack(float* f) const { Vec16<__nv_bfloat16>::unpack(v, f); }
};

// the same for four
template <typename T> struct Raw4;
template <> struct Raw4<float> {
    float4 v;
    __device__ __forceinline__ void load(const float* p) { v = *reinterpret_cast<const float4*>(p); }
    __device__ __forceinline__ void unpack(float* f) const { f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w; }
};
template <> struct Raw4<__nv_bfloat16> {
    uint2 v;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint2*>(p); }
    __device__ __forceinline__ void unpack(float* f) const {
        f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
        f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
    }
};

// out[r, :] = x[r, :] * inverse[r] * weight, inverse[r] = 1 / sqrt(mean(x[r, :]^2) + eps).  VEC: width a multiple of 8 and
// 32-byte aligned rows.
template <typename TX, typename TO, bool VEC>
__global__ void __launch_bounds__(kThreads)
rms_norm_kernel(const TX* __restrict__ x, const float* __restrict__ weight, TO* __restrict__ out, float* __restrict__ inverse,
                long long rows, long long width, float eps) {
    chain_begin();
    const int lane = threadIdx.x & 31;
    const long long warp = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5), nwarps = (long long)gridDim.x * kWarpsPerBlock;
    for (long long r = warp; r < rows; r += nwarps) {
        const TX* src = x + r * width;
        TO* dst = out + r * width;
        float total = 0.f;
        if (VEC) {
            for (long long c = lane * 8; c < width; c += 256) {
                float f[8];
                load8(src + c, f);
#pragma unroll
                for (int e = 0; e < 8; ++e) total = fmaf(f[e], f[e], total);
            }
        } else {
            for (long long c = lane; c < width; c += 32) {
                const float v = Act<TX>::load(src + c);
                total = fmaf(v, v, total);
            }
        }
        total = warp_sum(total);
        const float inv = rsqrtf(total / (float)width + eps);
        if (lane == 0) inverse[r] = inv;
        if (VEC) {
            for (long long c = lane * 8; c < width; c += 256) {
                float f[8], w[8];
                load8(src + c, f);
                load8(weight + c, w);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = f[e] * inv * w[e];
                store8(dst + c, f);
            }
        } else {
            for (long long c = lane; c < width; c += 32) Act<TO>::store(dst + c, Act<TX>::load(src + c) * inv * weight[c]);
        }
    }
}

// dx[r, c] = inv (g w - x inv^2 projected), projected = sum_c g w x / width   (lm_rms_dx, cpu_lm.py:84-104)
template <typename TG, typename TX, bool VEC>
__global__ void __launch_bounds__(kThreads)
rms_norm_dx_kernel(const TG* __restrict__ gradient, const TX* __restrict__ x, const float* __restrict__ weight,
                   const float* __restrict__ inverse, TX* __restrict__ dx, long long rows, long long width) {
    chain_begin();
    const int lane = threadIdx.x & 31;
    const long long warp = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5), nwarps = (long long)gridDim.x * kWarpsPerBlock;
    for (long long r = warp; r < rows; r += nwarps) {
        const TG* g = gradient + r * width;
        const TX* src = x + r * width;
        TX* dst = dx + r * width;
        float projected = 0.f;
        if (VEC) {
            for (long long c = lane * 8; c < width; c += 256) {
                float a[8], b[8], w[8];
                load8(g + c, a); load8(src + c, b); load8(weight + c, w);
#pragma unroll
                for (int e = 0; e < 8; ++e) projected = fmaf(a[e] * w[e], b[e], projected);
            }
        } else {
            for (long long c = lane; c < width; c += 32) projected = fmaf(Act<TG>::load(g + c) * weight[c], Act<TX>::load(src + c), projected);
        }
        projected = warp_sum(projected) / (float)width;
        const float inv = inverse[r];
        if (VEC) {
            for (long long c = lane * 8; c < width; c += 256) {
                float a[8], b[8], w[8];
                load8(g + c, a); load8(src + c, b); load8(weight + c, w);
#pragma unroll
                for (int e = 0; e < 8; ++e) a[e] = inv * (a[e] * w[e] - b[e] * inv * inv * projected);
                store8(dst + c, a);
            }
        } else {
            for (long long c = lane; c < width; c += 32)
                Act<TX>::store(dst + c, inv * (Act<TG>::load(g + c) * weight[c] - Act<TX>::load(src + c) * inv * inv * projected));
        }
    }
}

// partial[b, c] = sum over the rows of slab b of g[r, c] x[r, c] inverse[r]   (lm_rms_dw, one slab of rows per block).  VEC: a thread owns COLS
// neighbouring columns, and the rows are added in order, FLIGHT of them in flight (launch_dw_partial).
template <typename TG, typename TX, bool VEC, int COLS, int FLIGHT>
__global__ void __launch_bounds__(kThreads)
rms_norm_dw_partial_kernel(const TG* __restrict__ gradient, const TX* __restrict__ x, const float* __restrict__ inverse,
                           float* __restrict__ partial, long long rows, long long width) {
    chain_begin();
    const long long first = (long long)blockIdx.x * kSlabRows;
    const long long last = first + kSlabRows < rows ? first + kSlabRows : rows;
    if (VEC) {
        for (long long c = (long long)threadIdx.x * COLS; c < width; c += (long long)COLS * kThreads) {
            float total[COLS] = {};
            for (long long r0 = first; r0 < last; r0 += FLIGHT) {
                std::conditional_t<COLS == 8, Raw8<TG>, Raw4<TG>> g[FLIGHT];
                std::conditional_t<COLS == 8, Raw8<TX>, Raw4<TX>> v[FLIGHT];
                float inv[FLIGHT];
#pragma unroll
                for (int u = 0; u < FLIGHT; ++u) {
                    // past the slab's end: of four rows the last one again, left out of the sum below, so that no load waits for a test (fp32, 16384 x
                    // 2048, 161 us with one and 154); of more, nothing
                    const long long r = FLIGHT > 4 || r0 + u < last ? r0 + u : last - 1;
                    if (FLIGHT > 4 && r >= last) continue;
                    g[u].load(gradient + r * width + c);
                    v[u].load(x + r * width + c);
                    inv[u] = inverse[r];
                }
#pragma unroll
                for (int u = 0; u < FLIGHT; ++u)
                    if (r0 + u < last) {
                        float a[COLS], b[COLS];
                        g[u].unpack(a);
                        v[u].unpack(b);
#pragma unroll
                        for (int j = 0; j < COLS; ++j) total[j] = fmaf(a[j] * b[j], inv[u], total[j]);
                    }
            }
#pragma unroll
            for (int j = 0; j < COLS; j += 4)
                *reinterpret_cast<float4*>(partial + (long long)blockIdx.x * width + c + j) = make_float4(total[j], total[j + 1], total[j + 2], total[j + 3]);
        }
        return;
    }
    for (long long c = threadIdx.x; c < width; c += kThreads) {
        float total = 0.f;
        for (long long r = first; r < last; ++r)
            total = fmaf(Act<TG>::load(gradient + r * width + c) * Act<TX>::load(x + r * width + c), inverse[r], total);
        partial[(long long)blockIdx.x * width + c] = total;
    }
}
// out[c] = sum over the slabs, in order.  A block owns 32 columns; its eight warps take the slabs b = w, w + 8, ... and
// their sums are added in the order of w: the same tree on every run.
__global__ void __launch_bounds__(kThreads)
sum_partials_kernel(const float* __restrict__ partial, float* __restrict__ out, long long slabs, long long width) {
    chain_begin();
    __shared__ float part[kWarpsPerBlock][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (long long c0 = (long long)blockIdx.x * 32; c0 < width; c0 += (long long)gridDim.x * 32) {
        const long long c = c0 + lane;
        float total = 0.f;
        if (c < width)
            for (long long b = w; b < slabs; b += kWarpsPerBlock) total += partial[b * width + c];
        part[w][lane] = total;
        __syncthreads();
        if (w == 0 && c < width) {
            float sum = part[0][lane];
#pragma unroll
            for (int i = 1; i < kWarpsPerBlock; ++i) sum += part[i][lane];
            out[c] = sum;
        }
        __syncthreads();
    }
}

// Rotation of every pair (2 i, 2 i + 1) of every head by (offset + t) theta^(-2 i / dim)   (lm_rope, cpu_lm.py:125-138)
template <typename T>
__global__ void __launch_bounds__(kThreads)
rope_kernel(const T* __restrict__ values, T* __restrict__ out, long long pairs, int time, int heads, int dim, float theta,
            int offset, int inverse) {
    chain_begin();
    const int half = dim / 2;
    const float step = -2.f * log2f(theta) / (float)dim;
    for (long long i = (long long)blockIdx.x * kThreads + threadIdx.x; i < pairs; i += (long long)gridDim.x * kThreads) {
        const int j = (int)(i % half);
        const long long t = (i / half / heads) % time;
        float angle = (float)(offset + t) * exp2f(step * (float)j);
        if (inverse) angle = -angle;
        float s, c;
        sincosf(angle, &s, &c);
        const float a = Act<T>::load(values + 2 * i), b = Act<T>::load(values + 2 * i + 1);
        Act<T>::store(out + 2 * i, a * c - b * s);
        Act<T>::store(out + 2 * i + 1, a * s + b * c);
    }
}
// The same rotation with the angles of a position computed once for several heads: a thread owns (sequence, position, kRopeHeads
// heads, four neighbouring pairs = eight elements) and has its heads' loads in flight together.  dim a multiple of 8, rows on 32-byte boundaries.
// All heads in one thread, one after the other, left 602 positions to 19 blocks: 8 heads of 64 5.7 us, like this 2.6; 8192 positions, 16 and 4
// heads together 16.0 and 9.4.  More threads cost more angles: four heads share theirs.
constexpr int kRopeHeads = 4;
template <typename T>
__global__ void __launch_bounds__(kThreads)
rope_heads_kernel(const T* __restrict__ values, T* __restrict__ out, long long positions, int time, int heads, int dim, float theta,
                  int offset, int inverse) {
    chain_begin();
    const int groups = dim / 8, chunks = (heads + kRopeHeads - 1) / kRopeHeads;
    const float step = -2.f * log2f(theta) / (float)dim;
    for (long long i = (long long)blockIdx.x * kThreads + threadIdx.x; i < positions * chunks * groups; i += (long long)gridDim.x * kThreads) {
        const int group = (int)(i % groups), first = (int)(i / groups % chunks) * kRopeHeads;
        const long long position = i / groups / chunks, t = position % time;
        const long long base = position * heads * dim + 8 * group + (long long)first * dim;
        Raw8<T> raw[kRopeHeads];
#pragma unroll
        for (int h = 0; h < kRopeHeads; ++h)
            if (first + h < heads) raw[h].load(values + base + (long long)h * dim);
        float s[4], c[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float angle = (float)(offset + t) * exp2f(step * (float)(4 * group + q));
            if (inverse) angle = -angle;
            sincosf(angle, &s[q], &c[q]);
        }
#pragma unroll
        for (int h = 0; h < kRopeHeads; ++h) {
            if (first + h >= heads) break;
            float f[8], r[8];
            raw[h].unpack(f);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                r[2 * q] = f[2 * q] * c[q] - f[2 * q + 1] * s[q];
                r[2 * q + 1] = f[2 * q] * s[q] + f[2 * q + 1] * c[q];
            }
            store8(out + base + (long long)h * dim, r);
        }
    }
}

// out[i, :] = weight[ids[i], :]   (lm_embedding)
template <typename TO>
__global__ void __launch_bounds__(kThreads)
embedding_kernel(const float* __restrict__ weight, const long long* __restrict__ ids, TO* __restrict__ out, long long count,
                 long long width, long long vocab) {
    chain_begin();
    const int lane = threadIdx.x & 31;
    const long long warp = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5), nwarps = (long long)gridDim.x * kWarpsPerBlock;
    for (long long i = warp; i < count; i += nwarps) {
        const long long token = ids[i];
        const bool known = token >= 0 && token < vocab;     // an id outside the table reads nothing and gives a zero row
        for (long long c = lane; c < width; c += 32) Act<TO>::store(out + i * width + c, known ? weight[token * width + c] : 0.f);
    }
}

// d_weight[token[s], :] (+)= sum over the positions of segment s, in order, of gradient[position, :]
// (lm_embedding_backward: tokens sorted, each with the list of its positions)
template <typename TG, bool VEC>
__global__ void __launch_bounds__(kThreads)
embedding_backward_kernel(const TG* __restrict__ gradient, const long long* __restrict__ tokens, const long long* __restrict__ starts,
                          const long long* __restrict__ positions, float* __restrict__ d_weight, long long segments, long long width,
                          long long vocab, long long count, int parts) {
    chain_begin();
    // A warp owns (segment, part): columns [part * span, (part + 1) * span) of the token's row.
    // A frequent token has thousands of positions (Zipf-distributed ids put a third of a batch on one token); its
    // row is walked by `parts` warps side by side, each adding the positions in the order given, four rows in flight.
    const int lane = threadIdx.x & 31;
    const long long warp = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5), nwarps = (long long)gridDim.x * kWarpsPerBlock;
    const long long span = VEC ? 256 : width;   // the launch gives parts = ceil(width / 256) in the vector form, else 1
    for (long long item = warp; item < segments * parts; item += nwarps) {
        const long long s = item / parts, part = item - s * parts;
        const long long token = tokens[s];
        if (token < 0 || token >= vocab) continue;
        const long long begin = starts[s], end = starts[s + 1];
        const long long c_begin = part * span, c_end = c_begin + span < width ? c_begin + span : width;
        float* row = d_weight + token * width;
        if (VEC) {
            for (long long c = c_begin + lane * 8; c < c_end; c += 256) {
                float total[8];
                load8(row + c, total);
                long long at = begin;
                constexpr int kFlight = sizeof(TG) == 2 ? 16 : 8;     // rows in flight: 16 bytes (bf16) or 32 (fp32) per lane each
                for (; at + kFlight <= end; at += kFlight) {
                    Raw8<TG> raw[kFlight];
                    bool in[kFlight];
#pragma unroll
                    for (int u = 0; u < kFlight; ++u) {
                        const long long position = positions[at + u];
                        in[u] = position >= 0 && position < count;
                        if (in[u]) raw[u].load(gradient + position * width + c);
                    }
#pragma unroll
                    for (int u = 0; u < kFlight; ++u)
                        if (in[u]) {
                            float f[8];
                            raw[u].unpack(f);
#pragma unroll
                            for (int j = 0; j < 8; ++j) total[j] += f[j];
                        }
                }
                for (; at < end; ++at) {
                    const long long position = positions[at];
                    if (position < 0 || position >= count) continue;
                    float f[8];
                    load8(gradient + position * width + c, f);
#pragma unroll
                    for (int j = 0; j < 8; ++j) total[j] += f[j];
                }
                store8(row + c, total);
            }
        } else {
            for (long long c = c_begin + lane; c < c_end; c += 32) {
                float total = row[c];
                for (long long at = begin; at < end; ++at) {
                    const long long position = positions[at];
                    if (position >= 0 && position < count) total += Act<TG>::load(gradient + position * width + c);
                }
                row[c] = total;
            }
        }
    }
}

bool known_dtype(int dtype) { return dtype == QMOE_F32 || dtype == QMOE_BF16; }

}  // namespace
}  // namespace qmoe

using namespace qmoe;

extern "C" int qmoe_rms_norm(uint64_t x, int32_t x_dtype, uint64_t weight, uint64_t out, int32_t out_dtype, uint64_t inverse,
                             int64_t rows, int64_t width, double eps, uint64_t stream_) {
    if (!x || !weight || !out || !inverse) return fail_arg("rms_norm: null address");
    if (rows <= 0 || width <= 0) return fail_arg("rms_norm: sizes must be positive");
    if (!known_dtype(x_dtype) || !known_dtype(out_dtype)) return fail_arg("rms_norm: dtype must be QMOE_F32 or QMOE_BF16");
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_NORM, stream);
    const int grid = row_grid(rows);
    const float* w = (const float*)weight;
    float* inv = (float*)inverse;
    const bool vec = width % 8 == 0 && !((x | out | weight) & 31u);
#define QMOE_RMS_FORWARD(TX, TO)                                                                                               \
    do {                                                                                                                       \
        if (vec) chained(rms_norm_kernel<TX, TO, true>, grid, kThreads, 0, stream, (const TX*)x, w, (TO*)out, inv, rows, width, (float)eps);  \
        else chained(rms_norm_kernel<TX, TO, false>, grid, kThreads, 0, stream, (const TX*)x, w, (TO*)out, inv, rows, width, (float)eps);     \
    } while (0)
    if (x_dtype == QMOE_BF16 && out_dtype == QMOE_F32) QMOE_RMS_FORWARD(__nv_bfloat16, float);
    else if (x_dtype == QMOE_BF16) QMOE_RMS_FORWARD(__nv_bfloat16, __nv_bfloat16);
    else if (out_dtype == QMOE_F32) QMOE_RMS_FORWARD(float, float);
    else QMOE_RMS_FORWARD(float, __nv_bfloat16);
#undef QMOE_RMS_FORWARD
    QMOE_LAUNCH_CHECK("rms_norm_kernel");
    return 0;
}

// A slab of 32 rows is a chain of round trips to memory: the fewer slabs there are, the more rows of a slab have to be in flight, and with more slabs
// than SMs other blocks' loads are, and wide loads and few registers serve better.  Up to a slab for every SM: four columns per thread (twice the
// threads with work) and sixteen rows (8 of fp32), but eight columns where four take a second walk (width above 1024) or few rows are
// there to be had.  us for the whole backward with 4 columns x 16 rows, 8 x 8 and 8 x 4, bf16: 602 x 512 8.1, 8.3 and 9.7; 602 x 2048 13.6, 11.5 and 12.9; 4 x
// 1024 6.2, 5.7 and 5.6; 4096 x 1024 13.4, 13.6 and 15.0; 8192 x 512 17.9, 18.2 and 17.5; 16384 x 1024 47.0, 45.7 and 41.1; 32768 x 2048 170, 158 and 152.  fp32 with
// 4 x 8 and 8 x 4: 602 x 512 7.9 and 9.6; 8192 x 1024 34.2 and 36.3; 8192 x 2048 74.7 and 71.6.
template <typename TG, typename TX>
static void launch_dw_partial(bool vec, const TG* gradient, const TX* x, const float* inverse, float* partial, long long slabs, long long rows, long long width,
                       cudaStream_t stream) {
#define DW_PARTIAL(VEC, COLS, FLIGHT) chained(rms_norm_dw_partial_kernel<TG, TX, VEC, COLS, FLIGHT>, (unsigned)slabs, kThreads, 0, stream, gradient, x, inverse, partial, rows, width)
    constexpr bool HALF = sizeof(TG) + sizeof(TX) == 4;
    const bool many = slabs > sm_count();
    if (!vec) DW_PARTIAL(false, 4, 1);
    else if (HALF ? many : (many || rows <= 8) && width > 4 * kThreads) DW_PARTIAL(true, 8, 4);
    else if (HALF && (width > 4 * kThreads || rows <= 8)) DW_PARTIAL(true, 8, 8);
    else DW_PARTIAL(true, 4, (HALF ? 16 : 8));
#undef DW_PARTIAL
}

extern "C" int64_t qmoe_rms_norm_partials(int64_t rows, int64_t width) {
    return rows > 0 && width > 0 ? ((rows + kSlabRows - 1) / kSlabRows) * width : 0;
}

extern "C" int qmoe_rms_norm_backward(uint64_t gradient, int32_t g_dtype, uint64_t x, int32_t x_dtype, uint64_t weight,
                                      uint64_t inverse, uint64_t dx, uint64_t d_weight, uint64_t partials, int64_t rows,
                                      int64_t width, uint64_t stream_) {
    if (!gradient || !x || !weight || !inverse || !dx || !d_weight || !partials) return fail_arg("rms_norm_backward: null address");
    if (rows <= 0 || width <= 0) return fail_arg("rms_norm_backward: sizes must be positive");
    if (!known_dtype(g_dtype) || !known_dtype(x_dtype)) return fail_arg("rms_norm_backward: dtype must be QMOE_F32 or QMOE_BF16");
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_NORM, stream);
    const int grid = row_grid(rows);
    const long long slabs = (rows + kSlabRows - 1) / kSlabRows;
    const float* w = (const float*)weight;
    const float* inv = (const float*)inverse;
    float* part = (float*)partials;
    const bool vec = width % 8 == 0 && !((gradient | x | dx | weight | partials) & 31u);
#define QMOE_RMS_BACKWARD(TG, TX)                                                                                              \
    do {                                                                                                                       \
        if (vec) chained(rms_norm_dx_kernel<TG, TX, true>, grid, kThreads, 0, stream, (const TG*)gradient, (const TX*)x, w, inv, (TX*)dx, rows, width);   \
        else chained(rms_norm_dx_kernel<TG, TX, false>, grid, kThreads, 0, stream, (const TG*)gradient, (const TX*)x, w, inv, (TX*)dx, rows, width);      \
        launch_dw_partial(vec, (const TG*)gradient, (const TX*)x, inv, part, slabs, rows, width, stream);                                                 \
    } while (0)
    if (g_dtype == QMOE_BF16 && x_dtype == QMOE_BF16) QMOE_RMS_BACKWARD(__nv_bfloat16, __nv_bfloat16);
    else if (g_dtype == QMOE_BF16) QMOE_RMS_BACKWARD(__nv_bfloat16, float);
    else if (x_dtype == QMOE_BF16) QMOE_RMS_BACKWARD(float, __nv_bfloat16);
    else QMOE_RMS_BACKWARD(float, float);
#undef QMOE_RMS_BACKWARD
    QMOE_LAUNCH_CHECK("rms_norm_dx_kernel");
    chained(sum_partials_kernel, (unsigned)((width + 31) / 32), kThreads, 0, stream, part, (float*)d_weight, slabs, width);
    QMOE_LAUNCH_CHECK("sum_partials_kernel");
    return 0;
}

extern "C" int qmoe_rope(uint64_t values, uint64_t out, int32_t dtype, int64_t batch, int64_t time, int32_t heads, int32_t dim,
                         double theta, int32_t offset, int32_t inverse, uint64_t stream_) {
    if (!values || !out) return fail_arg("rope: null address");
    if (batch <= 0 || time <= 0 || heads <= 0 || dim <= 0 || dim % 2 || theta <= 0) return fail_arg("rope: sizes must be positive, dim even, theta positive");
    if (!known_dtype(dtype)) return fail_arg("rope: dtype must be QMOE_F32 or QMOE_BF16");
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_ELEMENTWISE, stream);
    const long long pairs = batch * time * heads * (dim / 2), positions = batch * time;
    const bool by_position = dim % 8 == 0 && !((values | out) & 31u);
    if (by_position && dtype == QMOE_BF16)
        chained(rope_heads_kernel<__nv_bfloat16>, flat_grid(positions * ((heads + kRopeHeads - 1) / kRopeHeads) * (dim / 8)), kThreads, 0, stream, (const __nv_bfloat16*)values, (__nv_bfloat16*)out, positions,
                                                                                     (int)time, heads, dim, (float)theta, offset, inverse);
    else if (by_position)
        chained(rope_heads_kernel<float>, flat_grid(positions * ((heads + kRopeHeads - 1) / kRopeHeads) * (dim / 8)), kThreads, 0, stream, (const float*)values, (float*)out, positions, (int)time,
                                                                                     heads, dim, (float)theta, offset, inverse);
    else if (dtype == QMOE_BF16)
        chained(rope_kernel<__nv_bfloat16>, flat_grid(pairs), kThreads, 0, stream, (const __nv_bfloat16*)values, (__nv_bfloat16*)out, pairs, (int)time, heads, dim,
                                                               (float)theta, offset, inverse);
    else
        chained(rope_kernel<float>, flat_grid(pairs), kThreads, 0, stream, (const float*)values, (float*)out, pairs, (int)time, heads, dim, (float)theta,
                                                               offset, inverse);
    QMOE_LAUNCH_CHECK("rope_kernel");
    return 0;
}

extern "C" int qmoe_embedding(uint64_t weight, uint64_t ids, uint64_t out, int32_t out_dtype, int64_t count, int64_t width,
                              int64_t vocab, uint64_t stream_) {
    if (!weight || !ids || !out) return fail_arg("embedding: null address");
    if (count <= 0 || width <= 0 || vocab <= 0) return fail_arg("embedding: sizes must be positive");
    if (!known_dtype(out_dtype)) return fail_arg("embedding: dtype must be QMOE_F32 or QMOE_BF16");
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_ELEMENTWISE, stream);
    if (out_dtype == QMOE_BF16)
        chained(embedding_kernel<__nv_bfloat16>, row_grid(count), kThreads, 0, stream, (const float*)weight, (const long long*)ids, (__nv_bfloat16*)out, count, width, vocab);
    else
        chained(embedding_kernel<float>, row_grid(count), kThreads, 0, stream, (const float*)weight, (const long long*)ids, (float*)out, count, width, vocab);
    QMOE_LAUNCH_CHECK("embedding_kernel");
    return 0;
}

// Host side of the embedding's backward: a counting sort over the vocabulary (interpreted, the tables of 8192 ids and their
// uploads were 2.0 of the 5.5 ms that a four-block training step takes to issue).
extern "C" int qmoe_token_tables(const void* ids_, int64_t count, int64_t vocab, void* distinct_, void* starts_, void* positions_, int64_t* segments) {
    if (!ids_ || !distinct_ || !starts_ || !positions_ || !segments) return fail_arg("token_tables: null address");
    if (count <= 0 || vocab <= 0) return fail_arg("token_tables: sizes must be positive");
    const int64_t* ids = (const int64_t*)ids_;
    int64_t *distinct = (int64_t*)distinct_, *starts = (int64_t*)starts_, *positions = (int64_t*)positions_;
    for (int64_t i = 0; i < count; ++i)
        if (ids[i] < 0 || ids[i] >= vocab) return fail_arg("token id outside the vocabulary");
    int64_t* next = (int64_t*)calloc((size_t)vocab, sizeof(int64_t));     // occurrences, then where the next position of a token goes
    if (!next) { set_error("token_tables: out of host memory"); return QMOE_ERR_STATE; }
    for (int64_t i = 0; i < count; ++i) ++next[ids[i]];
    int64_t found = 0, at = 0;
    for (int64_t t = 0; t < vocab; ++t) {
        const int64_t n = next[t];
        if (!n) continue;
        distinct[found] = t;
        starts[found++] = at;
        next[t] = at;
        at += n;
    }
    starts[found] = at;
    for (int64_t i = 0; i < count; ++i) positions[next[ids[i]]++] = i;
    free(next);
    *segments = found;
    return 0;
}

extern "C" int qmoe_embedding_backward(uint64_t gradient, int32_t g_dtype, uint64_t tokens, uint64_t starts, uint64_t positions,
                                       uint64_t d_weight, int64_t segments, int64_t count, int64_t width, int64_t vocab,
                                       uint64_t stream_) {
    if (!gradient || !tokens || !starts || !positions || !d_weight) return fail_arg("embedding_backward: null address");
    if (segments <= 0 || count <= 0 || width <= 0 || vocab <= 0) return fail_arg("embedding_backward: sizes must be positive");
    if (!known_dtype(g_dtype)) return fail_arg("embedding_backward: dtype must be QMOE_F32 or QMOE_BF16");
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_ELEMENTWISE, stream);
    // vector form: rows of 8-element pieces on 32-byte boundaries; spans of 256 columns per warp
    const bool vec = width % 8 == 0 && !((gradient | d_weight) & 31u);
    const int parts = vec ? (int)((width + 255) / 256) : 1;
    const int grid = row_grid(segments * parts);
#define QMOE_EMBEDDING_BACKWARD(TG, VEC)                                                                                              \
    chained(embedding_backward_kernel<TG, VEC>, grid, kThreads, 0, stream, (const TG*)gradient, (const long long*)tokens, (const long long*)starts, \
                                                                      (const long long*)positions, (float*)d_weight, segments, width, vocab, \
                                                                      count, parts)
    if (g_dtype == QMOE_BF16) {
        if (vec) QMOE_EMBEDDING_BACKWARD(__nv_bfloat16, true); else QMOE_EMBEDDING_BACKWARD(__nv_bfloat16, false);
    } else {
        if (vec) QMOE_EMBEDDING_BACKWARD(float, true); else QMOE_EMBEDDING_BACKWARD(float, false);
    }
#undef QMOE_EMBEDDING_BACKWARD
    QMOE_LAUNCH_CHECK("embedding_backward_kernel");
    return 0;
}
