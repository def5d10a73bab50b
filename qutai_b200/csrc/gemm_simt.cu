// CUDA-core GEMM (fp32 accumulate) used where the tensor-core path does not apply:
//  * the router (fp32 semantics whatever the activation dtype, skinny N = experts) and its backward;
//  * the expert FFN when activations are fp32 (the 1e-4 parity mode) or the widths are not
//    multiples of 8;
//  * the single-group `qmoe_gemm` of the host-side function table for shapes the tensor-core
//    kernel does not take.
// One generic kernel: arbitrary element strides for both operands, optional second (A2, B2) segment
// accumulated into the same tile, and three ways of grouping by expert.
#include <type_traits>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace qmoe {

namespace {

template <typename T> __device__ __forceinline__ float ldf(const T* p, long long i) { return Act<T>::load(p + i); }

template <typename TA, typename TB, typename TC, int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__(256)
simt_gemm_kernel(SimtGemmArgs g) {
    constexpr int BK = 16;
    static_assert((BM / TM) * (BN / TN) == 256, "256 threads");
    __shared__ float As[BK][BM + 4];
    __shared__ float Bs[BK][BN + 4];
    const int tid = threadIdx.x;
    const long long m0 = (long long)blockIdx.y * BM, n0 = (long long)blockIdx.x * BN;
    long long M = g.M, k_begin = 0, k_end = g.K;
    const TA* A = (const TA*)g.A;
    const TB* B = (const TB*)g.B;
    const TA* A2 = (const TA*)g.A2;
    const TB* B2 = (const TB*)g.B2;
    TC* C = (TC*)g.C;
    if (g.mode == SG_ROWS) {
        M = g.meta[0];
        if (m0 >= M) return;
        const long long e = g.tile_expert[m0 / kRowPad];
        B += e * g.b_slab;
        if (B2) B2 += e * g.b_slab;
    } else if (g.mode == SG_K) {
        const int e = blockIdx.z;
        if (g.counts[e] == 0) return;  // expert received nothing: its slab is left untouched
        k_begin = g.offsets[e];
        k_end = k_begin + g.counts[e];
        C += (long long)e * g.c_slab;
    } else if (g.mode == SG_SPLITK) {
        k_begin = (long long)blockIdx.z * g.k_chunk;
        k_end = k_begin + g.k_chunk < g.K ? k_begin + g.k_chunk : g.K;
        C += (long long)blockIdx.z * g.c_slab;
    }
    if (m0 >= M) return;

    const int tx = tid % (BN / TN), ty = tid / (BN / TN);
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    const bool a_kfast = g.a_cs == 1, b_kfast = g.b_rs == 1;
    for (int seg = 0; seg < 2; ++seg) {
        const TA* Ap = seg ? A2 : A;
        const TB* Bp = seg ? B2 : B;
        if (!Ap) break;
        for (long long k0 = k_begin; k0 < k_end; k0 += BK) {
#pragma unroll
            for (int l = 0; l < BM * BK / 256; ++l) {
                const int i = tid + l * 256;
                const int kk = a_kfast ? i % BK : i / BM;
                const int mm = a_kfast ? i / BK : i % BM;
                const long long m = m0 + mm, k = k0 + kk;
                As[kk][mm] = (m < M && k < k_end) ? ldf(Ap, m * g.a_rs + k * g.a_cs) : 0.f;
            }
#pragma unroll
            for (int l = 0; l < BN * BK / 256; ++l) {
                const int i = tid + l * 256;
                const int kk = b_kfast ? i % BK : i / BN;
                const int nn = b_kfast ? i / BK : i % BN;
                const long long n = n0 + nn, k = k0 + kk;
                Bs[kk][nn] = (n < g.N && k < k_end) ? ldf(Bp, k * g.b_rs + n * g.b_cs) : 0.f;
            }
            __syncthreads();
#pragma unroll
            for (int kk = 0; kk < BK; ++kk) {
                float a[TM], b[TN];
#pragma unroll
                for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
                for (int j = 0; j < TN; ++j) b[j] = Bs[kk][tx * TN + j];
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const long long m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const long long n = n0 + tx * TN + j;
            if (n >= g.N) continue;
            TC* dst = C + m * g.ldc + n;
            float v = acc[i][j];
            if (g.accumulate) v += Act<TC>::load(dst);
            Act<TC>::store(dst, v);
        }
    }
}

// ---- fp32 operands, many rows: 128 x 128 tiles, or 128 x 256 ------------------------------------------------------
// The same sums in the same order (one fp32 FMA chain per output, k ascending) as the kernel above, bit for bit; what
// differs is how the operands reach the FMAs.  That kernel fetches two shared-memory words for every four FMAs and
// stalls on each tile's loads (19 .. 25 TFLOP/s from 128 tiles on); here (30 .. 46) a thread owns 8 x 8 outputs (two 4-row and two 4-column pieces, so that
// the reads of a warp are whole 16-byte broadcasts), multiplies pairs of columns with one fma.rn.f32x2, and the next
// 16-deep tile travels from global memory through registers into the other shared buffer meanwhile.
// A_KFAST / B_KFAST: the operand is contiguous along k (rows of 4 k per load, transposed on the way into shared memory),
// else along its own rows / columns.
constexpr int TILE = 128, TILE_K = 16, WIDE = 256;

template <bool KFAST, int ROWS>
struct TileLoader {          // this thread's ROWS / 16 values of a TILE_K x ROWS slice of one operand
    const float* base;       // element (row 0 of the tile, k = 0)
    long long pitch;         // elements between rows (KFAST) or between k (not KFAST)
    int rows_left;           // rows of the tile inside the matrix
    static constexpr int PIECES = ROWS / 64;
    float v[4 * PIECES];
    __device__ __forceinline__ void fetch(long long k0, long long k_end) {
#pragma unroll
        for (int l = 0; l < PIECES; ++l) {
            const int i = threadIdx.x + l * 256;
            const int row = KFAST ? i / 4 : i % (ROWS / 4) * 4, k = KFAST ? i % 4 * 4 : i / (ROWS / 4);
            float* dst = v + 4 * l;
            const float* src = base + (KFAST ? row * pitch + (k0 + k) : (k0 + k) * pitch + row);
            const int along = KFAST ? (int)(k_end - (k0 + k) < 4 ? k_end - (k0 + k) : 4) : rows_left - row;   // values of the 4 that exist
            const bool across = KFAST ? row < rows_left : k0 + k < k_end;
            if (across && along >= 4) {
                const float4 w = *reinterpret_cast<const float4*>(src);
                dst[0] = w.x; dst[1] = w.y; dst[2] = w.z; dst[3] = w.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) dst[e] = across && e < along ? src[e] : 0.f;
            }
        }
    }
    __device__ __forceinline__ void store(float (*tile)[ROWS + 4]) const {
#pragma unroll
        for (int l = 0; l < PIECES; ++l) {
            const int i = threadIdx.x + l * 256;
            if (KFAST) {
#pragma unroll
                for (int e = 0; e < 4; ++e) tile[i % 4 * 4 + e][i / 4] = v[4 * l + e];
            } else {
                *reinterpret_cast<float4*>(&tile[i / (ROWS / 4)][i % (ROWS / 4) * 4]) = make_float4(v[4 * l], v[4 * l + 1], v[4 * l + 2], v[4 * l + 3]);
            }
        }
    }
};

// Products that share a launch: their tiles follow one another in blockIdx.x.  A product of 256 tiles leaves the last round of the
// 296 CTAs that are resident (two per SM) part empty; the three weight gradients together do so once.
struct SimtTileArgs {
    SimtGemmArgs product[kSimtProducts];
    int end[kSimtProducts];       // tiles of the products up to and including this one
    int columns[kSimtProducts];   // tiles side by side
};
template <bool ALONE> using TileArgs = std::conditional_t<ALONE, SimtGemmArgs, SimtTileArgs>;
__device__ __forceinline__ int product_index(const SimtGemmArgs&) { return 0; }
__device__ __forceinline__ int product_index(const SimtTileArgs& args) {
    const int tile = (int)blockIdx.x;
    return tile < args.end[0] ? 0 : tile < args.end[1] ? 1 : 2;
}
__device__ __forceinline__ const SimtGemmArgs& product_at(const SimtGemmArgs& args, int) { return args; }
__device__ __forceinline__ const SimtGemmArgs& product_at(const SimtTileArgs& args, int which) { return args.product[which]; }
template <int TN>
__device__ __forceinline__ void tile_at(const SimtGemmArgs&, int, long long& m0, long long& n0) {
    m0 = (long long)blockIdx.y * TILE;
    n0 = (long long)blockIdx.x * TN;
}
template <int TN>
__device__ __forceinline__ void tile_at(const SimtTileArgs& args, int which, long long& m0, long long& n0) {
    const int local = (int)blockIdx.x - (which ? args.end[which - 1] : 0);
    m0 = (long long)(local / args.columns[which]) * TILE;
    n0 = (long long)(local % args.columns[which]) * TN;
}

template <bool A_KFAST, bool B_KFAST, bool ALONE, int TN, int CTAS>
__global__ void __launch_bounds__(256, CTAS)
simt_tile_kernel(const __grid_constant__ TileArgs<ALONE> args) {
    const int which = product_index(args);
    const SimtGemmArgs& g = product_at(args, which);
    __shared__ __align__(16) float a_fixed[TN == TILE ? 2 : 1][TILE_K][TILE + 4];
    __shared__ __align__(16) float b_fixed[TN == TILE ? 2 : 1][TILE_K][TILE + 4];
    extern __shared__ __align__(16) float launch_memory[];         // the wide tiles' 50 KiB
    float (*const As)[TILE_K][TILE + 4] = TN == TILE ? a_fixed : reinterpret_cast<float (*)[TILE_K][TILE + 4]>(launch_memory);
    float (*const Bs)[TILE_K][TN + 4] = reinterpret_cast<float (*)[TILE_K][TN + 4]>(TN == TILE ? &b_fixed[0][0][0] : launch_memory + 2 * TILE_K * (TILE + 4));
    constexpr int GROUPS = TN / 64;       // four columns of every 64 are this thread's
    long long m0, n0;
    tile_at<TN>(args, which, m0, n0);
    long long M = g.M, k_begin = 0, k_end = g.K, b_offset = 0;
    float* C = (float*)g.C;
    if (g.mode == SG_ROWS) {
        M = g.meta[0];
        if (m0 >= M) return;
        b_offset = (long long)g.tile_expert[m0 / kRowPad] * g.b_slab;
    } else if (g.mode == SG_K) {
        const int e = blockIdx.z;
        if (g.counts[e] == 0) return;  // expert received nothing: its slab is left untouched
        k_begin = g.offsets[e];
        k_end = k_begin + g.counts[e];
        C += (long long)e * g.c_slab;
    }
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    uint64_t acc[8][2 * GROUPS];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 2 * GROUPS; ++j) acc[i][j] = 0ull;
    for (int seg = 0; seg < 2; ++seg) {
        const float* Ap = (const float*)(seg ? g.A2 : g.A);
        if (!Ap) break;
        const float* Bp = (const float*)(seg ? g.B2 : g.B) + b_offset;
        TileLoader<A_KFAST, TILE> a{Ap + m0 * g.a_rs, A_KFAST ? g.a_rs : g.a_cs, (int)(M - m0 < TILE ? M - m0 : TILE)};
        TileLoader<B_KFAST, TN> b{Bp + n0 * g.b_cs, B_KFAST ? g.b_cs : g.b_rs, (int)(g.N - n0 < TN ? g.N - n0 : TN)};
        a.fetch(k_begin, k_end);
        b.fetch(k_begin, k_end);
        __syncthreads();               // the segment before has been read out of the buffers
        a.store(As[0]);
        b.store(Bs[0]);
        __syncthreads();
        int buffer = 0;
        for (long long k0 = k_begin; k0 < k_end; k0 += TILE_K, buffer ^= 1) {
            const bool more = k0 + TILE_K < k_end;
            if (more) {
                a.fetch(k0 + TILE_K, k_end);
                b.fetch(k0 + TILE_K, k_end);
            }
#pragma unroll
            for (int kk = 0; kk < TILE_K; ++kk) {
                const float4 a0 = *reinterpret_cast<const float4*>(&As[buffer][kk][ty * 4]), a1 = *reinterpret_cast<const float4*>(&As[buffer][kk][64 + ty * 4]);
                const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
                uint64_t bv[2 * GROUPS];
#pragma unroll
                for (int q = 0; q < GROUPS; ++q) {
                    const ulonglong2 two = *reinterpret_cast<const ulonglong2*>(&Bs[buffer][kk][q * 64 + tx * 4]);
                    bv[2 * q] = two.x;
                    bv[2 * q + 1] = two.y;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint64_t twice = pair2(av[i], av[i]);
#pragma unroll
                    for (int j = 0; j < 2 * GROUPS; ++j) acc[i][j] = fma2(twice, bv[j], acc[i][j]);
                }
            }
            if (more) {
                a.store(As[buffer ^ 1]);
                b.store(Bs[buffer ^ 1]);
                __syncthreads();       // the one barrier of a tile: the other buffer is complete, and nobody reads this one any more
            }
        }
    }
    const bool vec = g.ldc % 4 == 0 && ((uintptr_t)C & 15u) == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const long long m = m0 + (i / 4) * 64 + ty * 4 + i % 4;
        if (m >= M) continue;
#pragma unroll
        for (int half = 0; half < GROUPS; ++half) {
            const long long n = n0 + half * 64 + tx * 4;
            float v[4];
            unpair2(acc[i][2 * half], v[0], v[1]);
            unpair2(acc[i][2 * half + 1], v[2], v[3]);
            float* dst = C + m * g.ldc + n;
            if (vec && n + 4 <= g.N) {
                *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n + e < g.N) dst[e] = v[e];
            }
        }
    }
}

// What the 128 x 128 kernel takes: fp32 operands and results, each operand contiguous along one of its axes with whole
// 16-byte pieces, no accumulation, more than 64 rows and columns (fewer are one tile of the general kernel, and half of the work
// here is on what does not exist: 40000 x 1024 x 16 columns 140 us there and 280 here, 32 columns 271 and 282, 64 columns 281
// and 281 .. 300), an inner size of at least one slice (9472 x 4 x 128: 8 us there, 10 here), and a tile for every second SM (with fewer, the four times smaller tiles of the general
// kernel spread better: 48 tiles with K = 512 take 66 us there and 66 .. 70 here, 64 tiles 66 and 59 .. 72, 128 tiles 113 and
// 61 .. 72).
bool tile_kernel_ok(const SimtGemmArgs& g, long long m_extent, int groups) {
    if (kernel_variant(QMOE_VARIANT_NO_FLOAT32_TILES)) return false;
    if (g.accumulate || (g.mode != SG_PLAIN && g.mode != SG_ROWS && g.mode != SG_K)) return false;
    const bool a_kfast = g.a_cs == 1, b_kfast = g.b_rs == 1;
    if ((!a_kfast && g.a_rs != 1) || (!b_kfast && g.b_cs != 1)) return false;
    const long long a_pitch = a_kfast ? g.a_rs : g.a_cs, b_pitch = b_kfast ? g.b_cs : g.b_rs;
    if (a_pitch % 4 || b_pitch % 4 || g.b_slab % 4) return false;
    if (((uintptr_t)g.A | (uintptr_t)g.B | (uintptr_t)g.A2 | (uintptr_t)g.B2) & 15u) return false;
    if (g.N <= 64 || m_extent <= 64 || (g.mode != SG_K && g.K < TILE_K)) return false;
    return (long long)ceil_div(g.N, TILE) * ceil_div(m_extent, TILE) * groups * 2 >= sm_count();
}

template <bool A_KFAST, bool B_KFAST, bool ALONE, int TN, int CTAS>
int launch_tile_kernel(const TileArgs<ALONE>& args, dim3 grid, cudaStream_t stream) {
    static bool configured[64] = {};          // per device
    constexpr int SMEM_BYTES = TN == TILE ? 0 : 2 * TILE_K * (TILE + 4 + TN + 4) * (int)sizeof(float);
    int dev = 0;
    QMOE_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail_arg("device ordinal beyond 63");
    if (SMEM_BYTES && !configured[dev]) {
        QMOE_CUDA(cudaFuncSetAttribute(simt_tile_kernel<A_KFAST, B_KFAST, ALONE, TN, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        configured[dev] = true;
    }
    // Ordinary launches, as for the general kernel: in a chain the CTAs are handed out while those of the kernel before leave, two
    // to some SMs and none to others, which costs kernels that are as long as their slowest SM more than the gap (2048
    // rows, 512 x 1024, 8 experts, forward and backward: 1038 us, in a chain 1113; 700 rows, 320 x 300, 4 experts, on the general kernel: 346 and 445).
    simt_tile_kernel<A_KFAST, B_KFAST, ALONE, TN, CTAS><<<grid, 256, SMEM_BYTES, stream>>>(args);
    QMOE_LAUNCH_CHECK("simt_tile_kernel");
    return 0;
}
// The forms of the kernel: tiles of 128 x 128, two to an SM (at 128 registers, which spills a little in some); one to an SM; tiles of 128 x 256
// (for a product by itself, see tile_form: A transposed comes by itself without the index, A as it is with it).
enum { TILES_TWO, TILES_ONE, TILES_WIDE };
template <bool A_KFAST, bool B_KFAST, bool ALONE>
int launch_tile_form(int form, const TileArgs<ALONE>& args, dim3 grid, cudaStream_t stream) {
    if constexpr (!(A_KFAST && B_KFAST)) {
        if constexpr (A_KFAST != ALONE)
            if (form == TILES_WIDE) return launch_tile_kernel<A_KFAST, B_KFAST, ALONE, WIDE, 1>(args, grid, stream);
        if (form == TILES_ONE) return launch_tile_kernel<A_KFAST, B_KFAST, ALONE, TILE, 1>(args, grid, stream);
    }
    return launch_tile_kernel<A_KFAST, B_KFAST, ALONE, TILE, 2>(args, grid, stream);
}

// Which form: two to an SM, except where the tiles of another are a single round.  An SM takes 3.05 units (128 x 128 tiles at the full rate of its
// FMA units, of which every form reaches two thirds) for two tiles, 1.8 for the one of two that a last round leaves it, 1.64 for one
// alone, 2.92 for a wide one: up to a tile for every SM one alone is through first, and up to two a wide one, if the wide ones are no more than SMs.  In more
// rounds the 4 % of the wide ones is less than what two CTAs gain that follow one another freely, or than a guess of the experts' tiles is
// off, so wide tiles are for plain products alone.  us as two to an SM, one and wide: g W 4096 x 1024 x 1024 200, 208 and 189; 1024 x 4096 x 2048 427, 405
// and 728; 640 x 640 x 2560 72, 68 and 120; weight gradients of 1024 rows, 4096 x 1024 194, 205 and 185; of 1500, 2048 x 776, 163, 155 and 271; A
// transposed, 6684 x 140 x 4020 169, and 172 wide.  x W^T does not spill, and two to an
// SM serve it best or nearly (4096 x 1024 x 1024 193, 209 and 191; 1024 x 4096 x 2048 409, 411 and 741).  The same bits in every form.  With a short
// inner size the results' way to memory is the work, which more and smaller tiles do better (weight gradients of 5 rows per expert, 64 x 3 x 1600 x 320, in a
// call of 1672 us: 1806 wide).
// Against all as two to an SM: 468 plain products 0.97 on average, at most 1.008; 330 layers of 64 .. 4096 rows, 4 .. 64 experts, forward and
// backward, 0.993 and at most 1.006 (with wide tiles in every number of rounds 0.991, but up to 1.09: 4096 rows, 1984 x 448, 16 experts, top 1, 1851 us and
// 2020).  2048 rows, 512 x 1024, 8 experts: 1021 and 998 us (dX 225 and 203, a tile for each SM).
constexpr long long kFormDepth = 128;
int tile_form(const SimtGemmArgs* products, int count, long long m_extent, int groups) {
    if (products[0].a_cs == 1 && products[0].b_rs == 1) return TILES_TWO;
    if ((products[0].mode == SG_K ? products[0].mean_rows : products[0].K) < kFormDepth) return TILES_TWO;
    const long long sms = sm_count();
    long long narrow = 0, wide = 0;      // by the largest guess of the rows
    for (int guess = 0; guess < 3; ++guess) {
        long long tiles = 0, tiles_wide = 0;
        for (int i = 0; i < count; ++i) {
            const long long rows = products[i].row_tiles[guess] ? products[i].row_tiles[guess] : ceil_div(m_extent > 0 ? m_extent : products[i].M, TILE);
            tiles += rows * ceil_div(products[i].N, TILE) * groups;
            tiles_wide += rows * ceil_div(products[i].N, WIDE) * groups;
        }
        if (tiles > narrow) { narrow = tiles; wide = tiles_wide; }
    }
    if (narrow <= sms) return TILES_ONE;
    return products[0].mode == SG_PLAIN && count == 1 && narrow <= 2 * sms && wide <= sms ? TILES_WIDE : TILES_TWO;
}

int launch_tiles_together(const SimtGemmArgs* products, int count, long long m_extent, int groups, cudaStream_t stream) {
    const int form = tile_form(products, count, m_extent, groups);
    SimtTileArgs args = {};
    long long tiles = 0;
    for (int i = 0; i < kSimtProducts; ++i) {
        if (i < count) {
            args.product[i] = products[i];
            args.columns[i] = ceil_div(products[i].N, form == TILES_WIDE ? WIDE : TILE);
            tiles += (long long)args.columns[i] * ceil_div(m_extent > 0 ? m_extent : products[i].M, TILE);
        }
        args.end[i] = (int)tiles;
    }
    if (tiles >= (1ll << 31)) return fail_arg("gemm: too many tiles");
    const SimtGemmArgs& g = products[0];
    const dim3 grid((unsigned)tiles, 1, (unsigned)groups);
    const bool a_kfast = g.a_cs == 1, b_kfast = g.b_rs == 1;
    if (a_kfast && b_kfast) return launch_tile_form<true, true, false>(form, args, grid, stream);
    if (a_kfast) return launch_tile_form<true, false, false>(form, args, grid, stream);
    if (b_kfast) return launch_tile_form<false, true, false>(form, args, grid, stream);
    return launch_tile_form<false, false, false>(form, args, grid, stream);
}

constexpr int kMaxGridY = 65535;      // of a launch

// m_extent 0: every product's own M.  Which products share a launch, or take that form of the kernel by themselves, was measured
// (medians of 15, all forms in one job): the index that finds a tile's product costs registers, and at 128 of them spills.  x W^T spills
// nothing without it, and two such products one after the other are faster than together (gate, up and down of 2048 rows, 1024 x 2048, 8
// experts, top 2: 1172 us, with the index 1262; a single 4096 x 1024 x 1024: 192 and 210).  So are single products with A transposed
// (2048 x 776 x 1500, B as it is 153 and 162, transposed 153 and 156).  Single products of plain A and B are not (dX and d_h; 2049 x 776 x
// 1500: 164 and 159), nor are the three weight gradients of a call (512 x 1024: 330 us one after the other, 299 together).  Forward and
// backward, 2048 rows, 8 experts, every product alone, every product with the index, and like this: 512 x 1024 1122, 1047 and 1026 us;
// 1024 x 2048 3474, 3498 and 3409; 512 rows, 1024 x 800, 16 experts 908, 824 and 822.
int launch_tiles(const SimtGemmArgs* products, int count, long long m_extent, int groups, cudaStream_t stream) {
    const bool a_kfast = products[0].a_cs == 1, b_kfast = products[0].b_rs == 1;
    bool alone = a_kfast ? b_kfast : count == 1;
    for (int i = 0; i < count; ++i) alone = alone && ceil_div(m_extent > 0 ? m_extent : products[i].M, TILE) <= kMaxGridY;
    if (!alone) return launch_tiles_together(products, count, m_extent, groups, stream);
    for (int i = 0; i < count; ++i) {
        const int form = tile_form(products + i, 1, m_extent, groups);
        const dim3 grid(ceil_div(products[i].N, form == TILES_WIDE ? WIDE : TILE), ceil_div(m_extent > 0 ? m_extent : products[i].M, TILE), groups);
        int rc;
        if (a_kfast) rc = launch_tile_form<true, true, true>(form, products[i], grid, stream);
        else if (b_kfast) rc = launch_tile_form<false, true, true>(form, products[i], grid, stream);
        else rc = launch_tile_form<false, false, true>(form, products[i], grid, stream);
        if (rc) return rc;
    }
    return 0;
}

// sum S partial [S][n] slabs in a fixed order
__global__ void __launch_bounds__(256)
reduce_partials_kernel(const float* __restrict__ partials, float* __restrict__ out, long long n, int splits) {
    chain_begin();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s = 0.f;
    for (int z = 0; z < splits; ++z) s += partials[(long long)z * n + i];
    out[i] = s;
}

template <typename TA, typename TB, typename TC>
int launch_typed(const SimtGemmArgs& g, long long m_extent, int groups, cudaStream_t stream) {
    if (g.N <= 16) {
        dim3 grid(ceil_div(g.N, 16), ceil_div(m_extent, 128), groups);
        simt_gemm_kernel<TA, TB, TC, 128, 16, 2, 4><<<grid, 256, 0, stream>>>(g);
    } else {
        dim3 grid(ceil_div(g.N, 64), ceil_div(m_extent, 64), groups);
        simt_gemm_kernel<TA, TB, TC, 64, 64, 4, 4><<<grid, 256, 0, stream>>>(g);
    }
    QMOE_LAUNCH_CHECK("simt_gemm_kernel");
    return 0;
}

}  // namespace

// dtype codes: QMOE_F32 / QMOE_BF16 for each of A, B, C.  m_extent = rows the grid must cover.
int launch_simt_gemm(const SimtGemmArgs& g, int a_dtype, int b_dtype, int c_dtype, long long m_extent,
                     int groups, cudaStream_t stream) {
    using bf = __nv_bfloat16;
    const int key = (a_dtype << 2) | (b_dtype << 1) | c_dtype;
    switch (key) {
        case 0:
            if (tile_kernel_ok(g, m_extent, groups)) return launch_tiles(&g, 1, m_extent, groups, stream);
            return launch_typed<float, float, float>(g, m_extent, groups, stream);
        case 1: return launch_typed<float, float, bf>(g, m_extent, groups, stream);
        case 2: return launch_typed<float, bf, float>(g, m_extent, groups, stream);
        case 3: return launch_typed<float, bf, bf>(g, m_extent, groups, stream);
        case 4: return launch_typed<bf, float, float>(g, m_extent, groups, stream);
        case 5: return launch_typed<bf, float, bf>(g, m_extent, groups, stream);
        case 6: return launch_typed<bf, bf, float>(g, m_extent, groups, stream);
        case 7: return launch_typed<bf, bf, bf>(g, m_extent, groups, stream);
    }
    return fail_arg("bad dtype combination");
}

int launch_simt_gemms(const SimtGemmArgs* g, int count, int a_dtype, int b_dtype, int c_dtype, int groups, cudaStream_t stream) {
    bool together = count <= kSimtProducts && a_dtype == QMOE_F32 && b_dtype == QMOE_F32 && c_dtype == QMOE_F32;
    for (int i = 0; together && i < count; ++i)
        together = tile_kernel_ok(g[i], g[i].M, groups) && (g[i].a_cs == 1) == (g[0].a_cs == 1) && (g[i].b_rs == 1) == (g[0].b_rs == 1);
    if (together) return launch_tiles(g, count, 0, groups, stream);
    for (int i = 0; i < count; ++i)
        if (int rc = launch_simt_gemm(g[i], a_dtype, b_dtype, c_dtype, g[i].M, groups, stream)) return rc;
    return 0;
}

int launch_reduce_partials(const float* partials, float* out, long long n, int splits, cudaStream_t stream) {
    chained(reduce_partials_kernel, ceil_div(n, 256), 256, 0, stream, partials, out, n, splits);
    QMOE_LAUNCH_CHECK("reduce_partials_kernel");
    return 0;
}

}  // namespace qmoe

namespace qmoe {
namespace {
// The tokens of the router's weight gradient are cut into ranges that run side by side and are added in a fixed order: an
// [experts, width] product has few tiles (8 experts of width 512: 8 of them, 251 us for 2048 tokens in one range, 18 in 16).
constexpr long long kRouterSplitTokens = 128, kRouterMaxSplits = 32;
long long router_splits(long long tokens) {    // at most this many; never fewer for more tokens
    const long long splits = (tokens + kRouterSplitTokens - 1) / kRouterSplitTokens;
    return splits > kRouterMaxSplits ? kRouterMaxSplits : splits;
}
long long router_split_tokens(long long tokens) { return (tokens + router_splits(tokens) - 1) / router_splits(tokens); }
}

int simt_router_logits(uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t scores, int64_t tokens, int64_t width,
                       int32_t experts, cudaStream_t stream) {
    TimedScope timed(KC_ROUTER_GEMM, stream);
    SimtGemmArgs g = {};
    g.A = (const void*)x; g.B = (const void*)w_router; g.C = (void*)scores;
    g.M = tokens; g.N = experts; g.K = width;
    g.a_rs = width; g.a_cs = 1;
    g.b_rs = 1; g.b_cs = width;  // B(k, n) = W[n, k]
    g.ldc = experts;
    g.mode = SG_PLAIN;
    return launch_simt_gemm(g, x_dtype, QMOE_F32, QMOE_F32, tokens, 1, stream);
}

long long simt_router_partials(int64_t tokens, int32_t experts, int64_t width) {
    return router_splits(tokens) * experts * width;
}

int simt_router_backward(uint64_t d_scores, uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t dx_router,
                         uint64_t d_w_router, uint64_t partials, int64_t tokens, int64_t width, int32_t experts,
                         cudaStream_t stream) {
    TimedScope timed(KC_ROUTER_GEMM, stream);
    if (dx_router) {  // [T, d] = d_scores[T, E] . W[E, d]
        SimtGemmArgs g = {};
        g.A = (const void*)d_scores; g.B = (const void*)w_router; g.C = (void*)dx_router;
        g.M = tokens; g.N = width; g.K = experts;
        g.a_rs = experts; g.a_cs = 1;
        g.b_rs = width; g.b_cs = 1;
        g.ldc = width;
        g.mode = SG_PLAIN;
        if (int rc = launch_simt_gemm(g, QMOE_F32, QMOE_F32, QMOE_F32, tokens, 1, stream)) return rc;
    }
    if (d_w_router) {  // [E, d] = d_scores^T[E, T] . x[T, d], split over tokens, reduced in fixed order
        if (!partials) return fail_arg("router_backward: scratch is null");
        const long long per_split = router_split_tokens(tokens);
        const int splits = (int)((tokens + per_split - 1) / per_split);
        SimtGemmArgs g = {};
        g.A = (const void*)d_scores; g.B = (const void*)x; g.C = (void*)partials;
        g.M = experts; g.N = width; g.K = tokens;
        g.a_rs = 1; g.a_cs = experts;  // A(m = e, k = t) = d_scores[t, e]
        g.b_rs = width; g.b_cs = 1;
        g.ldc = width;
        g.mode = SG_SPLITK;
        g.k_chunk = per_split;
        g.c_slab = (long long)experts * width;
        if (int rc = launch_simt_gemm(g, QMOE_F32, x_dtype, QMOE_F32, experts, splits, stream)) return rc;
        if (int rc = launch_reduce_partials((const float*)partials, (float*)d_w_router,
                                            (long long)experts * width, splits, stream)) return rc;
    }
    return 0;
}

}  // namespace qmoe
