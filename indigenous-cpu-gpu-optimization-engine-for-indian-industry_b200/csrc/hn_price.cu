// Revised-simplex pricing on the device: the per-iteration O(nnz + n) work of
// HyperNova's SimplexSolver (core/lp/simplex.cpp), over the matrix's device
// A^T. The basis factorisation (FTRAN/BTRAN) stays on the host.
//
//   hn_price_reduced_costs  rc = c - A^T y                    (compute_reduced_costs, :1225-1233)
//   hn_price_devex_update   alpha = A^T u; s = max |alpha_j| over nonbasic j;
//                           w_j = max(w_j, (alpha_j / s)^2)    (update_devex_weights, :1235-1271)
//   hn_price_select         Bland: first improving column;
//                           ranked: the k best by |rc_j|/sqrt(w_j), index
//                           ascending on ties                  (select_entering_variable,
//                                                               ranked_candidates, :1283-1361)
//   hn_price_columns        dense columns a_j of A             (extract_column, :25-35)
//
// A^T x sums each column's contributions in increasing row order, which is
// the order of SparseMatrix::transpose_multiply's and update_devex_weights's
// scatters, so reduced costs and Devex rows are bit-identical to the
// reference's. Selection compares integer keys (score bits, then index) in
// fixed trees, so its result does not depend on the order the blocks arrive in.
#include <algorithm>
#include <climits>

#include "hn_spmv.cuh"

namespace hn {
namespace {

constexpr int kPT = 256;
constexpr int kPriceBlocks = 148 * 4;

constexpr int W_BAD = 0;  // workspace select word: column indices out of range

struct EpiReducedCost {
    const double* cost;
    double* rc;
    __device__ __forceinline__ void operator()(int j, double s) const { rc[j] = cost[j] - s; }
};

// s = max over nonbasic j of |alpha_j| (std::max from 0.0, NaN-ignoring).
__global__ void __launch_bounds__(kPT) devex_scale_kernel(int64_t n, const double* __restrict__ alpha,
                                                          const int32_t* __restrict__ nonbasis,
                                                          double* __restrict__ partials,
                                                          unsigned* __restrict__ counter, double* __restrict__ out) {
    if (!after_previous()) return;
    __shared__ double sh[32];
    __shared__ bool last;
    double v = 0.0;
    for (int64_t j = blockIdx.x * (int64_t)kPT + threadIdx.x; j < n; j += (int64_t)gridDim.x * kPT)
        if (nonbasis[j] >= 0) v = fmax(v, fabs(alpha[j]));
    double r = block_max<kPT>(v, sh);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = r;
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double t = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += kPT) t = fmax(t, __ldcg(partials + i));
    r = block_max<kPT>(t, sh);
    if (threadIdx.x == 0) {
        *out = r;
        *counter = 0u;
    }
}

__global__ void __launch_bounds__(kPT) devex_apply_kernel(int64_t n, const double* __restrict__ alpha,
                                                          const int32_t* __restrict__ nonbasis,
                                                          const double* __restrict__ scale,
                                                          double* __restrict__ w) {
    if (!after_previous()) return;
    const double s = *scale;
    if (s == 0.0) return;
    for (int64_t j = blockIdx.x * (int64_t)kPT + threadIdx.x; j < n; j += (int64_t)gridDim.x * kPT) {
        if (nonbasis[j] < 0) continue;
        const double t = alpha[j] / s;
        const double q = t * t;
        if (q > w[j]) w[j] = q;
    }
}

struct PriceArgs {
    int64_t n;
    const double* rc;
    const double* w;
    const int32_t* nonbasis;
    const uint8_t* artificial;
    int phase1, maximize;
    double tol;
};

// What the choice reads of a column; loaded apart from its use, so that several are in flight.
struct Column {
    double rc, w;
    bool skip;
};
__device__ __forceinline__ Column load_column(const PriceArgs& a, int64_t j) {
    Column c{0.0, 1.0, true};
    if (j >= a.n) return c;
    c.skip = a.nonbasis[j] < 0 || (!a.phase1 && a.artificial && a.artificial[j]);
    c.rc = a.rc[j];
    if (a.w) c.w = a.w[j];
    return c;
}

// Improving nonbasic column (the filters of ranked_candidates and of the
// Bland scan); score = |rc_j| / sqrt(w_j) with w guarded to 1.
__device__ __forceinline__ bool eligible(const PriceArgs& a, const Column& c, double& score) {
    const double rc = a.maximize ? -c.rc : c.rc;
    if (c.skip || !(rc < -a.tol)) return false;
    double w = c.w;
    if (!(w > 0.0) || !isfinite(w)) w = 1.0;
    score = fabs(rc) / sqrt(w);
    return true;
}

__device__ __forceinline__ int64_t min_i64(int64_t a, int64_t b) { return a < b ? a : b; }
template <int THREADS>
__device__ __forceinline__ int64_t block_min_i64(int64_t v, int64_t* sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = min_i64(v, __shfl_down_sync(0xffffffffu, v, o));
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    int64_t r = INT64_MAX;
    if (wid == 0) {
        r = lane < THREADS / 32 ? sh[lane] : INT64_MAX;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r = min_i64(r, __shfl_down_sync(0xffffffffu, r, o));
    }
    return r;  // valid in thread 0
}

// A column of the ranking: score bits (scores are positive doubles, whose bit
// patterns order like their values; 0 = none) and index. Order: score
// descending, index ascending.
struct Pick {
    unsigned long long s, j;
};
__device__ __forceinline__ bool before(const Pick& a, const Pick& b) { return a.s > b.s || (a.s == b.s && a.j < b.j); }
// The warp's first pick, by word reductions (a butterfly of pairs takes twenty
// shuffles). Indices need their upper word only where n reaches 2^32 (wide).
__device__ __forceinline__ Pick warp_best(const Pick& v, bool wide) {
    const unsigned hi = static_cast<unsigned>(v.s >> 32), lo = static_cast<unsigned>(v.s);
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    bool c = hi == mh && lo == ml;
    unsigned jh = 0u;
    if (wide) {
        jh = __reduce_min_sync(0xffffffffu, c ? static_cast<unsigned>(v.j >> 32) : ~0u);
        c = c && static_cast<unsigned>(v.j >> 32) == jh;
    }
    const unsigned jl = __reduce_min_sync(0xffffffffu, c ? static_cast<unsigned>(v.j) : ~0u);
    return Pick{(unsigned long long)mh << 32 | ml, (unsigned long long)jh << 32 | jl};
}

constexpr int kSelT = 512;  // threads of the ranked selection
constexpr int kSelE = 8;    // picks a thread holds of a chunk
constexpr int kSelChunk = kSelT * kSelE;
static_assert(HN_PRICE_MAX_K <= kSelT && kSelT / 32 == 16, "ranked selection shape");

// The k first picks of the block's chunks (chunk c: picks c kSelChunk ..) into
// list (shared memory, k entries, none = 0). load(i0, key) fills a thread's
// kSelE picks of the chunk at i0. The list so far competes as one more pick of
// k threads. One barrier per place: every warp reduces the warps' bests itself.
template <class Load>
__device__ __forceinline__ void select_chunks(int64_t first, int64_t step, int64_t n, int k, bool wide, Pick* list,
                                              Pick (*sw)[16], Load load) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < k) list[tid] = Pick{0ull, ~0ull};
    __syncthreads();
    for (int64_t i0 = first; i0 < n; i0 += step) {
        Pick key[kSelE];
        load(i0, key);
        Pick held = tid < k ? list[tid] : Pick{0ull, ~0ull};
        const Pick last = list[k - 1];
        bool any = false;
#pragma unroll
        for (int e = 0; e < kSelE; ++e) any |= key[e].s != 0ull && before(key[e], last);
        if (!__syncthreads_or(any)) continue;  // nothing of this chunk places
        auto own_best = [&]() {
            Pick b = held;
#pragma unroll
            for (int e = 0; e < kSelE; ++e)
                if (before(key[e], b)) b = key[e];
            return b;
        };
        Pick own = own_best();  // changes only where a place was taken
        for (int r = 0; r < k; ++r) {
            Pick best = warp_best(own, wide);
            if (lane == 0) sw[r & 1][warp] = best;
            __syncthreads();
            best = warp_best(sw[r & 1][lane & 15], wide);
            if (tid == 0) list[r] = best;
            if (best.s == 0ull) {  // the rest of the list keeps what it had: none of it is left
                for (int q = r + tid; q < k; q += kSelT) list[q] = Pick{0ull, ~0ull};
                break;
            }
            if (own.s == best.s && own.j == best.j) {
                if (held.j == best.j) held.s = 0ull;
#pragma unroll
                for (int e = 0; e < kSelE; ++e)
                    if (key[e].j == best.j) key[e].s = 0ull;
                own = own_best();
            }
        }
        __syncthreads();
    }
}

// Ranked selection in one pass: each block keeps the k first columns of its
// chunks, the last block to finish merges the blocks' lists the same way. (A
// pass for the best score, one for its lowest index and a close per place took
// 300 us for 16 places of 500,000 columns; this takes 33.)
__global__ void __launch_bounds__(kSelT, 1) price_ranked_kernel(PriceArgs a, int k, Pick* lists,
                                                             unsigned long long* counts, unsigned* ticket,
                                                             int64_t* out) {
    if (!after_previous()) return;
    __shared__ Pick list[HN_PRICE_MAX_K];
    __shared__ Pick sw[2][16];
    __shared__ int64_t sh[32];
    __shared__ bool s_last;
    const int tid = threadIdx.x;
    const bool wide = a.n > (int64_t(1) << 32);
    int64_t cnt = 0;
    select_chunks(blockIdx.x * (int64_t)kSelChunk, gridDim.x * (int64_t)kSelChunk, a.n, k, wide, list, sw,
                  [&](int64_t i0, Pick* key) {
                      Column c[kSelE];
#pragma unroll
                      for (int e = 0; e < kSelE; ++e) c[e] = load_column(a, i0 + e * kSelT + tid);
#pragma unroll
                      for (int e = 0; e < kSelE; ++e) {
                          double sc;
                          const bool in = eligible(a, c[e], sc);
                          cnt += in;
                          key[e] = Pick{in ? (unsigned long long)__double_as_longlong(sc) : 0ull,
                                        (unsigned long long)(i0 + e * kSelT + tid)};
                      }
                  });
    cnt = block_sum_i64<kSelT>(cnt, sh);
    if (gridDim.x > 1) {
        if (tid < k) lists[blockIdx.x * k + tid] = list[tid];
        if (tid == 0) counts[blockIdx.x] = (unsigned long long)cnt;
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        const int64_t all = (int64_t)gridDim.x * k;
        select_chunks(0, kSelChunk, all, k, wide, list, sw, [&](int64_t i0, Pick* key) {
#pragma unroll
            for (int e = 0; e < kSelE; ++e) {
                const int64_t i = i0 + e * kSelT + tid;
                key[e] = Pick{0ull, ~0ull};
                if (i < all) key[e] = Pick{__ldcg(&lists[i].s), __ldcg(&lists[i].j)};
            }
        });
        cnt = tid < (int)gridDim.x ? (int64_t)__ldcg(counts + tid) : 0;
        cnt = block_sum_i64<kSelT>(cnt, sh);
    }
    if (tid == 0) {
        out[0] = cnt;
        *ticket = 0u;
    }
    if (tid < k) out[1 + tid] = list[tid].s ? (int64_t)list[tid].j : -1;
}

// Count of improving columns and the first one (Bland), the last block closing.
__global__ void __launch_bounds__(kPT) price_bland_kernel(PriceArgs a, unsigned long long* part, unsigned* ticket,
                                                          int64_t* out) {
    if (!after_previous()) return;
    __shared__ int64_t sh[32];
    __shared__ bool s_last;
    int64_t cnt = 0, first = INT64_MAX;
    for (int64_t j = blockIdx.x * (int64_t)kPT + threadIdx.x; j < a.n; j += (int64_t)gridDim.x * kPT) {
        double sc;
        if (eligible(a, load_column(a, j), sc)) {
            ++cnt;
            if (j < first) first = j;
        }
    }
    cnt = block_sum_i64<kPT>(cnt, sh);
    first = block_min_i64<kPT>(first, sh);
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = (unsigned long long)cnt;
        part[2 * blockIdx.x + 1] = (unsigned long long)first;
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    cnt = 0;
    first = INT64_MAX;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kPT) {
        cnt += (int64_t)__ldcg(part + 2 * b);
        const int64_t f = (int64_t)__ldcg(part + 2 * b + 1);
        if (f < first) first = f;
    }
    cnt = block_sum_i64<kPT>(cnt, sh);
    first = block_min_i64<kPT>(first, sh);
    if (threadIdx.x == 0) {
        out[0] = cnt;
        out[1] = first == INT64_MAX ? -1 : first;
        *ticket = 0u;
    }
}

// Column cols[r], rows [i0, i0 + kColRows) of slice blockIdx.x: zeros, then
// the entries that lie there (a row of A^T ascends). Columns outside [0, n)
// are left zero and counted in *bad.
constexpr int kColRows = 8192;
__global__ void __launch_bounds__(kPT) column_gather_kernel(int64_t m, int64_t n, int64_t k,
                                                            const int32_t* __restrict__ rpT,
                                                            const int32_t* __restrict__ ciT,
                                                            const double* __restrict__ valT,
                                                            const int64_t* __restrict__ cols, double* __restrict__ out,
                                                            unsigned long long* bad) {
    if (!after_previous()) return;
    __shared__ int64_t sh[32];
    const int64_t slices = m > 0 ? (m + kColRows - 1) / kColRows : 1;
    const int64_t r = blockIdx.x / slices, i0 = (blockIdx.x % slices) * kColRows;
    if (blockIdx.x == 0) {
        int64_t b = 0;
        for (int64_t q = threadIdx.x; q < k; q += kPT) b += cols[q] < 0 || cols[q] >= n;
        b = block_sum_i64<kPT>(b, sh);
        if (threadIdx.x == 0) *bad = (unsigned long long)b;
    }
    const int64_t j = cols[r];
    const int64_t i1 = i0 + kColRows < m ? i0 + kColRows : m;
    double* o = out + r * m;
    for (int64_t i = i0 + threadIdx.x; i < i1; i += kPT) o[i] = 0.0;
    if (j < 0 || j >= n) return;
    __syncthreads();
    for (int32_t e = rpT[j] + threadIdx.x; e < rpT[j + 1]; e += kPT) {
        const int32_t i = ciT[e];
        if (i >= i0 && i < i1) o[i] = valT[e];
    }
}

int price_grid(int64_t n) {
    const int64_t b = (n + kPT - 1) / kPT;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, kPriceBlocks));
}

}  // namespace
}  // namespace hn

using namespace hn;

extern "C" {

int hn_price_reduced_costs(const hn_csr* A, const double* y, const double* cost, double* rc, void* stream) {
    return guard("hn_price_reduced_costs", [&] {
        require_init();
        if (!A || !y || !cost || !rc) fail(HN_ERR_INVALID_ARG, "null argument");
        if (!A->has_t) fail(HN_ERR_INVALID_ARG, "matrix was created without its transpose");
        spmv_launch(spmv_mat(A, 1), y, EpiReducedCost{cost, rc}, as_stream(stream));
    });
}

int hn_price_devex_update(const hn_csr* A, const double* u, const int32_t* nonbasis, double* weights,
                          double* alpha, void* stream) {
    return guard("hn_price_devex_update", [&] {
        require_init();
        if (!A || !u || !nonbasis || !weights || !alpha) fail(HN_ERR_INVALID_ARG, "null argument");
        if (!A->has_t) fail(HN_ERR_INVALID_ARG, "matrix was created without its transpose");
        cudaStream_t s = as_stream(stream);
        Workspace& w = workspace(s);
        spmv_launch(spmv_mat(A, 1), u, EpiAxpby{1.0, 0.0, alpha}, s);
        const int g = price_grid(A->n);
        double* scale = w.partials + 4 * kMaxReduceBlocks;
        launch_next(devex_scale_kernel, g, kPT, 0, s, A->n, alpha, nonbasis, w.partials, w.counter, scale);
        launched("devex_scale_kernel");
        launch_next(devex_apply_kernel, g, kPT, 0, s, A->n, alpha, nonbasis, scale, weights);
        launched("devex_apply_kernel");
    });
}

int hn_price_select(int64_t n, const double* rc, const double* weights, const int32_t* nonbasis,
                    const uint8_t* artificial, int phase1, int maximize, double optimality_tol, int rule, int64_t k,
                    int64_t* out, void* stream) {
    return guard("hn_price_select", [&] {
        require_init();
        if (n < 0 || !out || (n > 0 && (!rc || !nonbasis))) fail(HN_ERR_INVALID_ARG, "bad arguments");
        if (rule != HN_PRICE_BLAND && rule != HN_PRICE_RANKED) fail(HN_ERR_INVALID_ARG, "unknown pricing rule");
        if (rule == HN_PRICE_RANKED && (k < 1 || k > HN_PRICE_MAX_K)) fail(HN_ERR_INVALID_ARG, "k out of range");
        cudaStream_t s = as_stream(stream);
        Workspace& w = workspace(s);
        const PriceArgs a{n, rc, weights, nonbasis, artificial, phase1, maximize, optimality_tol};
        if (rule == HN_PRICE_BLAND) {
            launch_next(price_bland_kernel, price_grid(n), kPT, 0, s, a, w.price, w.counter + 1, out);
            launched("price_bland_kernel");
            return;
        }
        const int64_t chunks = (n + kSelChunk - 1) / kSelChunk;
        const int g = (int)std::max<int64_t>(1, std::min<int64_t>(chunks, kPriceLists));
        launch_next(price_ranked_kernel, g, kSelT, 0, s, a, (int)k, reinterpret_cast<Pick*>(w.price),
                    w.price + 2 * kPriceLists * HN_PRICE_MAX_K, w.counter + 1, out);
        launched("price_ranked_kernel");
    });
}

int hn_price_columns(const hn_csr* A, int64_t k, const int64_t* cols, double* out, void* stream) {
    return guard("hn_price_columns", [&] {
        require_init();
        if (!A || k < 0 || (k > 0 && (!cols || !out))) fail(HN_ERR_INVALID_ARG, "bad arguments");
        if (!A->has_t) fail(HN_ERR_INVALID_ARG, "matrix was created without its transpose");
        if (k == 0) return;
        cudaStream_t s = as_stream(stream);
        Workspace& w = workspace(s);
        const int64_t slices = std::max<int64_t>(1, (A->m + kColRows - 1) / kColRows);
        if (k > INT32_MAX / slices) fail(HN_ERR_INVALID_ARG, "too many columns for one call");
        launch_next(column_gather_kernel, (unsigned)(k * slices), kPT, 0, s, A->m, A->n, k, A->rpT, A->ciT, A->valT,
                    cols, out, w.select + W_BAD);
        launched("column_gather_kernel");
        unsigned long long bad = 0;
        check_cuda(cudaMemcpyAsync(&bad, w.select + W_BAD, sizeof(bad), cudaMemcpyDeviceToHost, s), "D2H flag");
        check_cuda(cudaStreamSynchronize(s), "column gather sync");
        if (bad) fail(HN_ERR_INVALID_ARG, "column index out of range");
    });
}

}  // extern "C"
