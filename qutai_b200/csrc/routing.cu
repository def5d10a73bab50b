// Routing: softmax / top-k gating, per-expert counts, padded offsets, stable dispatch permutation,
// utilisation, auxiliary loss and the routing backward.  All tables are produced on the device
// with no host synchronisation and no floating-point atomics (results are run-to-run identical).
//
// Semantics follow `routing` / `routing_backward` of the upstream CPU path
// (src/qutai/backends/cpu_lm.py:204-276): experts are ranked by probability, equal values keep the
// lower expert index first, the k selected probabilities are renormalised to sum to one, and inside
// one expert the routed rows keep increasing (token, slot) order.
#include <limits.h>

#include "common.cuh"

namespace qmoe {

namespace {

// A warp per token row of a block: the ranking of a row is a serial chain (32768 rows, 64 experts, top 6: 57 us with four rows
// per warp and ten shuffles per slot, 27 like this).
constexpr int kWarps = 32;
static_assert(kWarps == kRouteRowsPerBlock, "one row per warp");
constexpr int kPackWarps = 8;
constexpr int kRowsPerPackWarp = kRouteRowsPerBlock / kPackWarps;

// Softmax and top-k of one token row by one warp; lane l holds experts l, l + 32, ... (EPL of them) of `scores`.  Lane s < k
// returns the expert and the gate weight of slot s; `p` are the row's probabilities.  Ranking uses the raw scores: softmax
// is strictly monotone, so this is the ranking by exact probability, without the extra ties that rounding the
// probabilities to fp32 would create.
template <int EPL>
__device__ __forceinline__ void rank_row(const float* __restrict__ scores, int E, int k, float (&p)[EPL], int& expert, float& weight) {
    const int lane = threadIdx.x & 31;
    float v[EPL], m = -INFINITY, s = 0.f;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        const int e = lane + 32 * j;
        v[j] = e < E ? scores[e] : -INFINITY;
        m = fmaxf(m, v[j]);
    }
    m = warp_max(m);
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        p[j] = lane + 32 * j < E ? expf(v[j] - m) : 0.f;
        s += p[j];
    }
    s = warp_sum(s);
    // top-k by (score descending, expert index ascending) over unsigned keys in the order of the scores (-0 counts as 0), so
    // that a slot is two warp reductions of one instruction each.  A NaN score ranks as -inf; the probabilities and gate
    // weights still carry the NaN to the output.  Key 0: no expert, or already taken.
    unsigned key[EPL];
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        p[j] = p[j] / s;
        const float score = v[j] != v[j] ? -INFINITY : v[j] + 0.f;
        const unsigned bits = __float_as_uint(score);
        key[j] = lane + 32 * j < E ? bits ^ ((unsigned)((int)bits >> 31) | 0x80000000u) : 0u;
    }
    float total = 0.f;
    expert = 0;
    weight = 0.f;
#pragma unroll
    for (int slot = 0; slot < kMaxTopK; ++slot) {
        if (slot >= k) break;
        unsigned best = key[0];
        int at = lane;
#pragma unroll
        for (int j = 1; j < EPL; ++j)
            if (key[j] > best) { best = key[j]; at = lane + 32 * j; }
        const unsigned top = __reduce_max_sync(0xffffffffu, best);
        const int winner = (int)__reduce_min_sync(0xffffffffu, best == top ? (unsigned)at : 0x7fffffffu);   // < E: k <= E
        float mine = 0.f;
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
            if (j == (winner >> 5)) mine = p[j];
            if (lane + 32 * j == winner) key[j] = 0u;
        }
        const float pw = __shfl_sync(0xffffffffu, mine, winner & 31);
        total += pw;  // left-to-right sum over the slots, like the upstream `sum(...)`
        if (lane == slot) { expert = winner; weight = pw; }
    }
    weight = weight / total;
}

// ---- K1: softmax + top-k + per-block histogram and probability column sums --------------------
template <int EPL>
__global__ void __launch_bounds__(kWarps * 32)
route_topk_kernel(const float* __restrict__ scores, float* __restrict__ probs,
                  float* __restrict__ gate_w, int* __restrict__ expert_idx,
                  int* __restrict__ block_counts, float* __restrict__ block_colsum,
                  long long T, int E, int k, int* __restrict__ row_source, long long rows_bound) {
    chain_begin();
    // every dispatched row a pad row until the packing kernel, two launches on, says otherwise; a memset between two kernels is a gap of 2 us on
    // both sides of its own 1.4
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < rows_bound; i += (long long)gridDim.x * blockDim.x) row_source[i] = -1;
    __shared__ int s_cnt[kMaxExperts];
    __shared__ float s_col[kWarps][32 * EPL];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < E; i += blockDim.x) s_cnt[i] = 0;
    __syncthreads();
    const long long row = (long long)blockIdx.x * kRouteRowsPerBlock + warp;
    float p[EPL];
#pragma unroll
    for (int j = 0; j < EPL; ++j) p[j] = 0.f;
    if (row < T) {
        int expert;
        float weight;
        rank_row<EPL>(scores + row * E, E, k, p, expert, weight);
        if (lane < k) {
            expert_idx[row * k + lane] = expert;
            gate_w[row * k + lane] = weight;
            atomicAdd(&s_cnt[expert], 1);  // integer: order does not matter
        }
#pragma unroll
        for (int j = 0; j < EPL; ++j)
            if (lane + 32 * j < E) probs[row * E + lane + 32 * j] = p[j];
    }
#pragma unroll
    for (int j = 0; j < EPL; ++j) s_col[warp][lane + 32 * j] = p[j];
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) t += s_col[w][e];  // fixed order
        block_colsum[(long long)blockIdx.x * E + e] = t;
        block_counts[(long long)blockIdx.x * E + e] = s_cnt[e];
    }
}

// ---- what follows from the counts and the probability sums of all experts -----------------------
// Two warps: the first forms the padded offsets (s_off) and writes meta, the second the auxiliary loss.  Fixed order.
__device__ __forceinline__ void publish_totals(const int* s_cnt, const double* s_cs, int* s_off, int* __restrict__ offsets, int* __restrict__ meta,
                                               float* __restrict__ aux, long long T, int E, int k) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        int before = 0;
        for (int base = 0; base < E; base += 32) {
            const int e = base + lane;
            const int padded = e < E ? (s_cnt[e] + kRowPad - 1) / kRowPad * kRowPad : 0;
            int sum = padded;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += up;
            }
            if (e < E) {
                s_off[e] = before + sum - padded;
                offsets[e] = before + sum - padded;
            }
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) {
            s_off[E] = before;
            offsets[E] = before;
            meta[0] = before;
            meta[1] = before / kRowPad;
            meta[2] = (int)(T * k);
            meta[3] = 0;
        }
    } else if (warp == 1) {
        const double A = (double)T * k;
        double total = 0.0;
        for (int e = lane; e < E; e += 32) total += ((double)s_cnt[e] / A) * s_cs[e] / (double)T;
#pragma unroll
        for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        if (lane == 0) aux[0] = (float)((double)E * total);
    }
}

// ---- K2: scan over blocks, padded offsets, tile map, utilisation and auxiliary loss -----------
// One block of 1024 threads: thread (segment, expert) first totals its segment of token blocks, the
// segments are prefixed per expert, then each thread writes the running bases of its segment.  All
// sums run in a fixed order (column sums in double), so the results are run-to-run identical.
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads)
route_scan_kernel(const int* __restrict__ block_counts, const float* __restrict__ block_colsum,
                  int* __restrict__ block_base, int* __restrict__ counts, int* __restrict__ offsets,
                  int* __restrict__ tile_expert, int* __restrict__ meta, float* __restrict__ util,
                  float* __restrict__ aux, int nblk, long long T, int E, int k) {
    chain_begin();
    __shared__ int s_seg[kScanThreads];
    __shared__ double s_segcs[kScanThreads];
    __shared__ int s_cnt[kMaxExperts];
    __shared__ int s_off[kMaxExperts + 1];
    __shared__ double s_cs[kMaxExperts];
    const int nseg = kScanThreads / E;
    const int seg = threadIdx.x / E, e = threadIdx.x - seg * E;
    const bool active = seg < nseg;
    const int chunk = (nblk + nseg - 1) / nseg;
    const int b0 = seg * chunk, b1 = min(nblk, b0 + chunk);
    if (active) {
        int total = 0;
        double cs = 0.0;
        for (int b = b0; b < b1; ++b) {
            total += block_counts[(long long)b * E + e];
            cs += (double)block_colsum[(long long)b * E + e];
        }
        s_seg[threadIdx.x] = total;
        s_segcs[threadIdx.x] = cs;
    }
    __syncthreads();
    if (active) {
        int run = 0;
        for (int s = 0; s < seg; ++s) run += s_seg[s * E + e];
        for (int b = b0; b < b1; ++b) {
            const int c = block_counts[(long long)b * E + e];
            block_base[(long long)b * E + e] = run;
            run += c;
        }
        if (seg == 0) {
            int total = 0;
            double cs = 0.0;
            for (int s = 0; s < nseg; ++s) { total += s_seg[s * E + e]; cs += s_segcs[s * E + e]; }
            counts[e] = total;
            s_cnt[e] = total;
            s_cs[e] = cs;
        }
    }
    __syncthreads();
    publish_totals(s_cnt, s_cs, s_off, offsets, meta, aux, T, E, k);
    __syncthreads();
    if (threadIdx.x < E) {
        const int x = threadIdx.x;
        util[x] = (float)((double)s_cnt[x] / ((double)T * k));
        for (int t = s_off[x] / kRowPad; t < s_off[x + 1] / kRowPad; ++t) tile_expert[t] = x;
    }
}

// ---- K3: stable rank of every assignment inside (block, expert) -> dispatch tables -----------
// Same block partition as K1.  Warp w owns a contiguous slice of the block's assignments; a
// `match_any` per 32-assignment chunk ranks equal experts by lane, so order is (token, slot).
__global__ void __launch_bounds__(kPackWarps * 32)
route_pack_kernel(const int* __restrict__ expert_idx, const int* __restrict__ block_base,
                  const int* __restrict__ offsets, int* __restrict__ dest_row,
                  int* __restrict__ row_source, long long T, int E, int k) {
    chain_begin();
    __shared__ int s_hist[kPackWarps][kMaxExperts];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kPackWarps * kMaxExperts; i += blockDim.x) (&s_hist[0][0])[i] = 0;
    __syncthreads();
    const long long A = T * k;
    const long long begin = ((long long)blockIdx.x * kRouteRowsPerBlock + warp * kRowsPerPackWarp) * k;
    long long end = begin + (long long)kRowsPerPackWarp * k;
    if (end > A) end = A;
    const unsigned lt = (1u << lane) - 1u;
    for (long long base = begin; base < end; base += 32) {
        const long long a = base + lane;
        const int e = a < end ? expert_idx[a] : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, e);
        if (e >= 0 && (peers & lt) == 0) s_hist[warp][e] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        int run = offsets[e] + block_base[(long long)blockIdx.x * E + e];
#pragma unroll
        for (int w = 0; w < kPackWarps; ++w) {
            const int c = s_hist[w][e];
            s_hist[w][e] = run;
            run += c;
        }
    }
    __syncthreads();
    for (long long base = begin; base < end; base += 32) {
        const long long a = base + lane;
        const int e = a < end ? expert_idx[a] : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, e);
        int dest = -1;
        if (e >= 0) dest = s_hist[warp][e] + __popc(peers & lt);
        __syncwarp();
        if (e >= 0 && (peers & lt) == 0) s_hist[warp][e] += __popc(peers);
        __syncwarp();
        if (e >= 0) {
            dest_row[a] = dest;
            row_source[dest] = (int)a;
        }
    }
}

// counts to pinned host memory
__global__ void publish_counts_kernel(const int* __restrict__ counts, int* __restrict__ host, int experts) {
    chain_begin();
    for (int e = threadIdx.x; e < experts; e += blockDim.x) host[e] = counts[e];
}

// ---- few tokens (decoding): the whole routing in one block -------------------------------------------
// At 64 tokens the three kernels above and the fill of row_source are four launches of which none has work for more than
// one or two SMs; here the same steps meet at block barriers (64 tokens, 64 experts, top 6: 31 us in four launches with one
// warp per four rows, 11 here; 4 tokens, 8 experts, top 2: 19 and 5.5).  What is left is the chain of a row's reductions.  A warp ranks the rows warp, warp + 32, ...; then warp w
// holds the w-th slice of at most 32 consecutive assignments, ranked among equals by `match_any`.
constexpr long long kSmallRouteTokens = 128;
static_assert(kSmallRouteTokens * kMaxTopK <= kWarps * 32, "a slice of assignments is one per lane");
template <int EPL>
__device__ __forceinline__ void route_small(const float* scores, float* __restrict__ probs, float* __restrict__ gate_w, int* __restrict__ expert_idx,
                                            int* __restrict__ dest_row, int* row_source, int* __restrict__ counts, int* __restrict__ offsets,
                                            int* __restrict__ tile_expert, int* __restrict__ meta, float* __restrict__ util, float* __restrict__ aux,
                                            float* __restrict__ block_colsum, int T, int E, int k, long long rows_bound) {
    // [warp][expert]: probability sums, then assignments; one more column, so that a warp reading one expert's 32 entries
    // meets 32 banks
    __shared__ union { float col[kWarps][32 * EPL + 1]; int hist[kWarps][32 * EPL + 1]; } s;
    __shared__ int s_idx[kSmallRouteTokens * kMaxTopK];
    __shared__ int s_cnt[32 * EPL], s_off[32 * EPL + 1];
    __shared__ double s_cs[32 * EPL];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (long long i = threadIdx.x; i < rows_bound; i += blockDim.x) row_source[i] = -1;
    float col[EPL];
#pragma unroll
    for (int j = 0; j < EPL; ++j) col[j] = 0.f;
    for (int row = warp; row < T; row += kWarps) {
        float p[EPL], weight;
        int expert;
        rank_row<EPL>(scores + (long long)row * E, E, k, p, expert, weight);
        if (lane < k) {
            s_idx[row * k + lane] = expert;
            expert_idx[row * k + lane] = expert;
            gate_w[row * k + lane] = weight;
        }
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
            col[j] += p[j];
            if (lane + 32 * j < E) probs[(long long)row * E + lane + 32 * j] = p[j];
        }
    }
#pragma unroll
    for (int j = 0; j < EPL; ++j) s.col[warp][lane + 32 * j] = col[j];
    __syncthreads();
    for (int e = warp; e < E; e += kWarps) {       // a warp per expert, its lanes the 32 partial sums
        double t = (double)s.col[lane][e];
#pragma unroll
        for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) s_cs[e] = t;
        // readers of the per-block sums (expert parallelism) add them over the blocks: the first holds all
        if (lane * kRouteRowsPerBlock < T) block_colsum[(long long)lane * E + e] = lane ? 0.f : (float)t;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kWarps * (32 * EPL + 1); i += blockDim.x) (&s.hist[0][0])[i] = 0;
    __syncthreads();
    const int A = T * k, slice = (A + kWarps - 1) / kWarps, a = warp * slice + lane;
    const int mine = lane < slice && a < A ? s_idx[a] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, mine);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    if (mine >= 0 && rank == 0) s.hist[warp][mine] = __popc(peers);
    __syncthreads();
    for (int e = warp; e < E; e += kWarps) {       // prefix over the slices
        const int own = s.hist[lane][e];
        int run = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += up;
        }
        s.hist[lane][e] = run - own;
        if (lane == 31) {
            s_cnt[e] = run;
            counts[e] = run;
            util[e] = (float)((double)run / (double)A);
        }
    }
    __syncthreads();
    publish_totals(s_cnt, s_cs, s_off, offsets, meta, aux, T, E, k);
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x)
        for (int t = s_off[e] / kRowPad; t < s_off[e + 1] / kRowPad; ++t) tile_expert[t] = e;
    if (mine >= 0) {
        const int dest = s_off[mine] + s.hist[warp][mine] + rank;
        dest_row[a] = dest;
        row_source[dest] = a;      // after the fill above: barriers lie between
    }
}

template <int EPL>
__global__ void __launch_bounds__(kWarps * 32, 1)
route_small_kernel(const float* __restrict__ scores, float* __restrict__ probs, float* __restrict__ gate_w, int* __restrict__ expert_idx,
                   int* __restrict__ dest_row, int* row_source, int* __restrict__ counts, int* __restrict__ offsets,
                   int* __restrict__ tile_expert, int* __restrict__ meta, float* __restrict__ util, float* __restrict__ aux,
                   float* __restrict__ block_colsum, int T, int E, int k, long long rows_bound) {
    chain_begin();
    route_small<EPL>(scores, probs, gate_w, expert_idx, dest_row, row_source, counts, offsets, tile_expert, meta, util, aux, block_colsum, T, E, k, rows_bound);
}

// The logits of a handful of tokens and their routing in one launch, a warp per logit.  us a call, in two launches and one: 4 rows, 8 experts,
// 1024 x 2816, norm to residual, called step by step 45.2 and 42.7 (its launches bound the host), the device alone 38.9 and 39.1; replayed without the
// norm 33.1 and 33.0, 1 row, 32 experts, 2048 x 1408, 41.2 .. 42.0 and 41.1, 1 row, 8 experts, 512 x 264, 22.6 and 20.6.  A second logit per warp is a second round trip: 8 rows, 8 experts, 39.8 and 41.5, 2 rows, 32 experts, 41.9 and 45.0.
constexpr int kRouterRouteLogits = kWarps;
template <typename X, bool NORM>
__global__ void __launch_bounds__(kWarps * 32, 1)
router_route_small_kernel(const X* __restrict__ x, const float* __restrict__ w, long long d, const float* __restrict__ norm_weight, float eps,
                          float* __restrict__ inverse, float* scores, float* __restrict__ probs, float* __restrict__ gate_w, int* __restrict__ expert_idx,
                          int* __restrict__ dest_row, int* row_source, int* __restrict__ counts, int* __restrict__ offsets,
                          int* __restrict__ tile_expert, int* __restrict__ meta, float* __restrict__ util, float* __restrict__ aux,
                          float* __restrict__ block_colsum, int T, int E, int k, long long rows_bound) {
    chain_begin();
    const int i = threadIdx.x >> 5;
    if (i < T * E) {
        const int t = i / E, e = i - t * E;
        float inv = 0.f;
        const float logit = small_logit<X, NORM>(x + t * d, w + e * d, d, norm_weight, eps, inv);
        if ((threadIdx.x & 31) == 0) {
            scores[i] = logit;
            if (NORM && e == 0) inverse[t] = inv;
        }
    }
    __syncthreads();        // the block reads its own logits
    route_small<1>(scores, probs, gate_w, expert_idx, dest_row, row_source, counts, offsets, tile_expert, meta, util, aux, block_colsum, T, E, k, rows_bound);
}

__global__ void route_export_kernel(const int* __restrict__ expert_idx, const int* __restrict__ dest_row,
                                    const int* __restrict__ offsets, const int* __restrict__ counts,
                                    long long* indices, long long* ids, long long* slots,
                                    long long* locations, long long* counts64, long long A, int E,
                                    int k, long long capacity) {
    chain_begin();
    const long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (a < E && counts64) counts64[a] = counts[a];
    if (a >= A) return;
    const int e = expert_idx[a];
    const long long loc = dest_row[a] - offsets[e];
    if (indices) indices[a] = e;
    if (locations) locations[a] = loc;
    if (ids) ids[e * capacity + loc] = a / k;
    if (slots) slots[e * capacity + loc] = a % k;
}

// ---- routing backward: one warp per token row -------------------------------------------------
__global__ void __launch_bounds__(256)
route_backward_kernel(const float* __restrict__ probs, const float* __restrict__ gate_w,
                      const int* __restrict__ expert_idx, const float* __restrict__ util,
                      const float* __restrict__ grad_w, const float* __restrict__ grad_aux,
                      float* __restrict__ d_scores, long long T, int E, int k) {
    chain_begin();
    const int lane = threadIdx.x & 31;
    const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= T) return;
    const float ga = grad_aux ? grad_aux[0] * (float)E / (float)T : 0.f;
    float center_aux = 0.f;
    if (grad_aux) {
        for (int e = lane; e < E; e += 32) center_aux += probs[row * E + e] * util[e];
        center_aux = warp_sum(center_aux);
    }
    float center = 0.f;
    if (grad_w)
        for (int s = 0; s < k; ++s) center += grad_w[row * k + s] * gate_w[row * k + s];
    for (int e = lane; e < E; e += 32) {
        float value = 0.f;
        if (grad_aux) value = ga * probs[row * E + e] * (util[e] - center_aux);
        if (grad_w)
            for (int s = 0; s < k; ++s)
                if (expert_idx[row * k + s] == e)
                    value += gate_w[row * k + s] * (grad_w[row * k + s] - center);
        d_scores[row * E + e] = value;
    }
}

// need_scratch: the three block tables are only used while the routing itself runs (qmoe_route); every
// consumer of a finished route accepts null there, so a route filled by qmoe_route_static can be passed on.
int check_route(const qmoe_route_t* r, bool need_scratch) {
    if (!r) return fail_arg("route is null");
    if (r->tokens <= 0) return fail_arg("tokens must be positive (got %lld)", (long long)r->tokens);
    if (r->experts <= 0 || r->experts > kMaxExperts)
        return fail_arg("experts must be in [1, %d] (got %d)", kMaxExperts, r->experts);
    // top_k <= experts is a property of routing.  The consumers of a finished route also take the expert-side view an
    // expert-parallel rank builds of its local experts, which can be fewer than top_k (8 experts top-2 over 8 ranks).
    if (r->top_k <= 0 || r->top_k > kMaxTopK || (need_scratch && r->top_k > r->experts))
        return fail_arg("top_k must be in [1, min(experts, %d)] (got %d)", kMaxTopK, r->top_k);
    if (r->tokens * r->top_k > (1ll << 30)) return fail_arg("tokens * top_k exceeds 2^30");
    if (r->rows_bound < qmoe_rows_bound(r->tokens, r->experts, r->top_k))
        return fail_arg("rows_bound %lld is smaller than qmoe_rows_bound()", (long long)r->rows_bound);
    if (!r->probs || !r->gate_weights || !r->expert_index || !r->dest_row || !r->row_source ||
        !r->counts || !r->offsets || !r->tile_expert || !r->meta || !r->utilization || !r->aux)
        return fail_arg("route has a null table address");
    if (need_scratch && (!r->block_counts || !r->block_base || !r->block_colsum))
        return fail_arg("route has a null scratch table address (block_counts / block_base / block_colsum)");
    return 0;
}

}  // namespace

int route_check(const qmoe_route_t* r) { return check_route(r, false); }

}  // namespace qmoe

using namespace qmoe;

extern "C" int64_t qmoe_rows_bound(int64_t tokens, int32_t experts, int32_t top_k) {
    const int64_t a = tokens * top_k + (int64_t)experts * (kRowPad - 1);
    return (a + kRowPad - 1) / kRowPad * kRowPad;
}

extern "C" int64_t qmoe_route_blocks(int64_t tokens) {
    return (tokens + kRouteRowsPerBlock - 1) / kRouteRowsPerBlock;
}

extern "C" int qmoe_route(const qmoe_route_t* r, uint64_t scores, uint64_t stream_) {
    if (int rc = check_route(r, true)) return rc;
    if (!scores) return fail_arg("scores is null");
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_ROUTE, stream);
    const int nblk = (int)qmoe_route_blocks(r->tokens);
    const long long T = r->tokens;
    const int E = r->experts, k = r->top_k;
    const float* sc = (const float*)scores;
    float* probs = (float*)r->probs;
    float* gw = (float*)r->gate_weights;
    int* eidx = (int*)r->expert_index;
    int* bc = (int*)r->block_counts;
    float* bs = (float*)r->block_colsum;
    const int epl = (E + 31) / 32;
    if (T <= kSmallRouteTokens) {
#define ARGS 1, kWarps * 32, 0, stream, sc, probs, gw, eidx, (int*)r->dest_row, (int*)r->row_source, (int*)r->counts, (int*)r->offsets, \
        (int*)r->tile_expert, (int*)r->meta, (float*)r->utilization, (float*)r->aux, bs, (int)T, E, k, (long long)r->rows_bound
        if (epl <= 1) chained(route_small_kernel<1>, ARGS);
        else if (epl <= 2) chained(route_small_kernel<2>, ARGS);
        else if (epl <= 4) chained(route_small_kernel<4>, ARGS);
        else chained(route_small_kernel<8>, ARGS);
#undef ARGS
        QMOE_LAUNCH_CHECK("route_small_kernel");
        return 0;
    }
    if (epl <= 1) chained(route_topk_kernel<1>, nblk, kWarps * 32, 0, stream, sc, probs, gw, eidx, bc, bs, T, E, k, (int*)r->row_source, (long long)r->rows_bound);
    else if (epl <= 2) chained(route_topk_kernel<2>, nblk, kWarps * 32, 0, stream, sc, probs, gw, eidx, bc, bs, T, E, k, (int*)r->row_source, (long long)r->rows_bound);
    else if (epl <= 4) chained(route_topk_kernel<4>, nblk, kWarps * 32, 0, stream, sc, probs, gw, eidx, bc, bs, T, E, k, (int*)r->row_source, (long long)r->rows_bound);
    else chained(route_topk_kernel<8>, nblk, kWarps * 32, 0, stream, sc, probs, gw, eidx, bc, bs, T, E, k, (int*)r->row_source, (long long)r->rows_bound);
    QMOE_LAUNCH_CHECK("route_topk_kernel");
    chained(route_scan_kernel, 1, kScanThreads, 0, stream, bc, bs, (int*)r->block_base, (int*)r->counts,
                                                      (int*)r->offsets, (int*)r->tile_expert,
                                                      (int*)r->meta, (float*)r->utilization,
                                                      (float*)r->aux, nblk, T, E, k);
    QMOE_LAUNCH_CHECK("route_scan_kernel");
    chained(route_pack_kernel, nblk, kPackWarps * 32, 0, stream, eidx, (const int*)r->block_base,
                                                        (const int*)r->offsets, (int*)r->dest_row,
                                                        (int*)r->row_source, T, E, k);
    QMOE_LAUNCH_CHECK("route_pack_kernel");
    return 0;
}

bool qmoe::router_route_ok(const qmoe_route_t* r) { return r->tokens <= kSmallRouteTokens && r->experts <= 32 && r->tokens * r->experts <= kRouterRouteLogits; }

int qmoe::router_route_small(const qmoe_route_t* r, uint64_t x, int32_t x_dtype, uint64_t w_router, uint64_t norm_weight, double eps, uint64_t inverse,
                             uint64_t scores, int64_t width, uint64_t stream_) {
    if (int rc = check_route(r, true)) return rc;
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_ROUTE, stream);
#define LAUNCH(X, NORM)                                                                                                                    \
    chained(router_route_small_kernel<X, NORM>, 1, kWarps * 32, 0, stream, (const X*)x, (const float*)w_router, (long long)width,          \
            (const float*)norm_weight, (float)eps, (float*)inverse, (float*)scores, (float*)r->probs, (float*)r->gate_weights,             \
            (int*)r->expert_index, (int*)r->dest_row, (int*)r->row_source, (int*)r->counts, (int*)r->offsets, (int*)r->tile_expert,        \
            (int*)r->meta, (float*)r->utilization, (float*)r->aux, (float*)r->block_colsum, (int)r->tokens, r->experts, r->top_k, (long long)r->rows_bound)
    if (x_dtype == QMOE_BF16) { if (norm_weight) LAUNCH(__nv_bfloat16, true); else LAUNCH(__nv_bfloat16, false); }
    else { if (norm_weight) LAUNCH(float, true); else LAUNCH(float, false); }
#undef LAUNCH
    QMOE_LAUNCH_CHECK("router_route_small_kernel");
    return 0;
}

extern "C" int qmoe_publish_counts(uint64_t counts, void* host, int32_t experts, uint64_t event, uint64_t stream_) {
    if (!counts || !host) return fail_arg("publish_counts: null address");
    if (experts <= 0) return fail_arg("publish_counts: experts must be positive");
    cudaStream_t stream = (cudaStream_t)stream_;
    chained(publish_counts_kernel, 1, experts < 256 ? (experts + 31) / 32 * 32 : 256, 0, stream, (const int*)counts, (int*)host, experts);
    QMOE_LAUNCH_CHECK("publish_counts_kernel");
    if (event) QMOE_CUDA(cudaEventRecord((cudaEvent_t)event, stream));
    return 0;
}

extern "C" int qmoe_route_export_i64(const qmoe_route_t* r, uint64_t indices, uint64_t ids, uint64_t slots,
                                     uint64_t locations, uint64_t counts, int64_t capacity,
                                     uint64_t stream_) {
    if (int rc = check_route(r, false)) return rc;
    const long long A = r->tokens * r->top_k;
    if ((ids || slots) && capacity < A) return fail_arg("capacity %lld is smaller than tokens*top_k", (long long)capacity);
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_OTHER, stream);
    const long long n = A > r->experts ? A : r->experts;
    chained(route_export_kernel, ceil_div(n, 256), 256, 0, stream, 
        (const int*)r->expert_index, (const int*)r->dest_row, (const int*)r->offsets,
        (const int*)r->counts, (long long*)indices, (long long*)ids, (long long*)slots,
        (long long*)locations, (long long*)counts, A, r->experts, r->top_k, capacity);
    QMOE_LAUNCH_CHECK("route_export_kernel");
    return 0;
}

extern "C" int qmoe_route_backward(const qmoe_route_t* r, uint64_t grad_weights, uint64_t grad_aux,
                                   uint64_t d_scores, uint64_t stream_) {
    if (int rc = check_route(r, false)) return rc;
    if (!d_scores) return fail_arg("d_scores is null");
    cudaStream_t stream = (cudaStream_t)stream_;
    TimedScope timed(KC_ROUTE_BWD, stream);
    if (!grad_weights && !grad_aux) {
        QMOE_CUDA(cudaMemsetAsync((void*)d_scores, 0, (size_t)r->tokens * r->experts * sizeof(float), stream));
        return 0;
    }
    chained(route_backward_kernel, ceil_div(r->tokens, 8), 256, 0, stream, 
        (const float*)r->probs, (const float*)r->gate_weights, (const int*)r->expert_index,
        (const float*)r->utilization, (const float*)grad_weights, (const float*)grad_aux,
        (float*)d_scores, r->tokens, r->experts, r->top_k);
    QMOE_LAUNCH_CHECK("route_backward_kernel");
    return 0;
}

// ---------------------------------------------------------------------------------------------
// qmoe_route_static: qmoe_route for callers that cannot supply scratch memory.
//
// qmoe_route needs three scratch tables (block_counts, block_base, block_colsum) besides its inputs
// and outputs, and expects the caller to allocate them.  Some hosts cannot: a serving loop that
// must never call cudaMalloc on its request path (the call synchronises the whole device), a
// plug-in host that was handed a fixed set of buffers at start-up and has no allocator of its own
// to reach for more, or a runtime whose memory pool is private to it.  For them the three tables
// live in the fixed device array below, which every GPU that loads this library keeps resident
// until the process exits (1.5 MiB).  The caller still passes every input and output table.
//
// Limit: blocks * experts <= kStaticRouteEntries, where blocks = qmoe_route_blocks(tokens); larger
// problems are rejected with an argument error and must use qmoe_route.
//
// The array is shared by all calls and keeps whatever the previous call left in it.  That is
// harmless here because the first routing kernel writes every entry it later reads (one row per
// block, all experts), so nothing has to start at zero and nothing is cleared.  It also means two
// calls whose kernels overlap on the GPU (different streams, or different host threads) race on the
// array: issue calls to this entry point on one stream at a time per device.
//
// The first call on a device looks up the array's device address (cudaGetSymbolAddress, checked)
// with that device current, and remembers it; make that first call before starting any stream
// capture.  The remembered address is written without a lock: two host threads that make the first
// call at the same moment both look the address up and store the same value.  No cudaMalloc, cudaFree or allocating library routine is called on any path.
namespace {
constexpr long long kStaticRouteEntries = 131072;  // entries per table (blocks * experts)
static __device__ __align__(256) unsigned char g_route_scratch[3 * kStaticRouteEntries * 4];
constexpr int kMaxDevices = 64;
void* g_route_scratch_address[kMaxDevices] = {nullptr};  // device address per device, looked up once
}  // namespace

extern "C" int qmoe_route_static(const qmoe_route_t* r, uint64_t scores, uint64_t stream_) {
    if (!r) return fail_arg("route is null");
    if (r->tokens <= 0 || r->experts <= 0) return fail_arg("route_static: tokens and experts must be positive");
    const long long entries = qmoe_route_blocks(r->tokens) * (long long)r->experts;
    if (entries > kStaticRouteEntries)
        return fail_arg("route_static: %lld blocks x %d experts = %lld scratch entries exceed the built-in %lld; "
                        "use qmoe_route with caller-allocated scratch",
                        (long long)qmoe_route_blocks(r->tokens), r->experts, entries, kStaticRouteEntries);
    int device = 0;
    QMOE_CUDA(cudaGetDevice(&device));
    if (device < 0 || device >= kMaxDevices) return fail_arg("route_static: device index %d is out of range", device);
    if (!g_route_scratch_address[device]) {
        // In host code `g_route_scratch` only stands for the symbol; the address kernels can use
        // has to be asked for, once per device, while that device is current.
        void* address = nullptr;
        QMOE_CUDA(cudaGetSymbolAddress(&address, g_route_scratch));
        if (!address) { set_error("route_static: the scratch array has no device address"); return QMOE_ERR_STATE; }
        g_route_scratch_address[device] = address;
    }
    unsigned char* base = (unsigned char*)g_route_scratch_address[device];
    qmoe_route_t with_scratch = *r;
    with_scratch.block_counts = (uint64_t)base;
    with_scratch.block_base = (uint64_t)(base + kStaticRouteEntries * 4);
    with_scratch.block_colsum = (uint64_t)(base + 2 * kStaticRouteEntries * 4);
    return qmoe_route(&with_scratch, scores, stream_);
}
