// Merge-path FP64 CSR SpMV with a fused per-row epilogue.
//
// The merge path is the interleaving of the m row ends (rp[1..m]) with the
// nnz nonzero indices; it is cut into tiles of kSpmvTile items so every CTA
// does the same amount of work whatever the row-length distribution (the
// Zipf-skewed A^T rows of the large configuration and the Poisson rows of A
// alike). Inside a tile each thread walks kSpmvIpt consecutive items.
//
// Per tile: the row ends go to shared memory; each thread finds where the
// path enters and leaves its items (two binary searches), loads the products
// of its contiguous nonzeros straight into registers (col_idx, values, then
// the x gathers -- through L1, so a warp's neighbouring ranges share sectors),
// and walks its items, finishing rows that end in its range; partial rows are
// combined through a shared carry array in thread order. A row that
// began in an earlier tile leaves its in-tile part in head_val and is
// finished by a second, tiny kernel that adds the earlier tiles' carries in
// tile order. Every row's sum therefore has a fixed association order, so
// results are deterministic run to run.
//
// Epilogues receive (row, sum) exactly once per row and write the outputs
// (y = alpha*s + beta*y, residuals, IPM directions ...).
#pragma once

#include "hn_internal.cuh"

namespace hn {

constexpr int kSpmvThreads = 256;
constexpr int kSpmvIpt = 7;
constexpr int kSpmvTile = kSpmvThreads * kSpmvIpt;

struct SpmvMat {
    int m, nnz;
    const int32_t* rp;
    const int32_t* ci;
    const double* val;
    const int32_t* tile_row;
    const int32_t* tile_nz;
    int32_t* carry_row;
    double* carry_val;
    int32_t* head_row;
    double* head_val;
    int64_t ntiles;
    int kind = 0;  // 0: merge path; 1: binned vector CSR
    const int32_t* perm = nullptr;
    SpmvBins bins = {};
    // the one-launch product (small_tile): tiles done of the running product,
    // zero in between (null: two launches), or, with short_heads, not needed
    unsigned* ticket = nullptr;
    bool short_heads = false;
};

inline SpmvMat spmv_mat(const hn_csr* A, int trans) {
    SpmvMat M;
    if (!trans) {
        M = SpmvMat{(int)A->m, (int)A->nnz, A->rp, A->ci, A->val, A->tile_row, A->tile_nz,
                    A->carry_row, A->carry_val, A->head_row, A->head_val, A->ntiles};
    } else {
        M = SpmvMat{(int)A->n, (int)A->nnz_t, A->rpT, A->ciT, A->valT, A->tile_row_t, A->tile_nz_t,
                    A->carry_row_t, A->carry_val_t, A->head_row_t, A->head_val_t, A->ntiles_t};
    }
    M.ticket = reinterpret_cast<unsigned*>(M.carry_row + M.ntiles);
    const int d = trans ? 1 : 0;
    M.short_heads = A->short_heads[d];
    if (A->spmv_kind[d] == 1 && A->perm[d]) {
        M.kind = 1;
        M.perm = A->perm[d];
        M.bins = A->bins[d];
    }
    return M;
}

// Merge-path coordinate of tile-local diagonal `diag`: rows consumed (return)
// and nonzeros consumed (diag - return), from the tile's row ends in shared memory.
__device__ __forceinline__ int tile_search(const int32_t* s_rowend, int k0, int diag, int nrows_t, int nnz_t) {
    int lo = diag - nnz_t > 0 ? diag - nnz_t : 0;
    int hi = diag < nrows_t ? diag : nrows_t;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (s_rowend[mid] <= k0 + diag - mid - 1)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

template <class Epi>
__global__ void __launch_bounds__(kSpmvThreads) spmv_tile_kernel(SpmvMat a, const double* __restrict__ x,
                                                                 Epi epi) {
    if (!after_previous()) return;
    __shared__ int32_t s_rowend[kSpmvTile + 1];
    __shared__ int32_t s_crow[kSpmvThreads];
    __shared__ double s_cval[kSpmvThreads];
    __shared__ int32_t s_rowstart0;

    const int tid = threadIdx.x;
    const int tile = blockIdx.x;
    const int r0 = a.tile_row[tile], k0 = a.tile_nz[tile];
    const int r1 = a.tile_row[tile + 1], k1 = a.tile_nz[tile + 1];
    const int nrows_t = r1 - r0;
    const int nnz_t = k1 - k0;

    if (tid == 0) {
        s_rowstart0 = (r0 < a.m) ? a.rp[r0] : a.nnz;
        a.head_row[tile] = -1;
    }
    for (int i = tid; i <= nrows_t; i += kSpmvThreads) {
        const int r = r0 + i;
        s_rowend[i] = (r < a.m) ? __ldg(a.rp + r + 1) : INT_MAX;
    }
    __syncthreads();

    // this thread's kSpmvIpt merge items: its nonzeros are the contiguous
    // range [nz, nz_e) of the tile, found from the path at both ends
    const int total_t = nrows_t + nnz_t;
    const int diag = min(tid * kSpmvIpt, total_t);
    const int diag_end = min(diag + kSpmvIpt, total_t);
    int row = tile_search(s_rowend, k0, diag, nrows_t, nnz_t);
    int nz = diag - row;
    const int row_e = tile_search(s_rowend, k0, diag_end, nrows_t, nnz_t);
    const int cnt = (diag_end - row_e) - nz;

    // products of those nonzeros, straight into registers (no shared buffer):
    // column indices first, then values, then the gathers of x
    double v[kSpmvIpt];
    {
        int c[kSpmvIpt];
#pragma unroll
        for (int u = 0; u < kSpmvIpt; ++u) c[u] = (u < cnt) ? __ldg(a.ci + k0 + nz + u) : 0;
        double w[kSpmvIpt];
#pragma unroll
        for (int u = 0; u < kSpmvIpt; ++u) w[u] = (u < cnt) ? __ldg(a.val + k0 + nz + u) : 0.0;
#pragma unroll
        for (int u = 0; u < kSpmvIpt; ++u) v[u] = (u < cnt) ? w[u] * __ldcg(x + c[u]) : 0.0;
    }

    double sum = 0.0;
    int first_row = -1;
    double first_val = 0.0;
#pragma unroll
    for (int it = 0; it < kSpmvIpt; ++it) {
        if (diag + it < diag_end) {
            const bool take_nz = (nz < nnz_t) && (k0 + nz < s_rowend[row]);
            if (take_nz) {
                sum += v[0];
#pragma unroll
                for (int q = 0; q < kSpmvIpt - 1; ++q) v[q] = v[q + 1];
                ++nz;
            } else if (row < nrows_t) {
                if (first_row < 0) {
                    first_row = row;
                    first_val = sum;
                } else {
                    epi(r0 + row, sum);
                }
                sum = 0.0;
                ++row;
            }
        }
    }
    s_crow[tid] = row;
    s_cval[tid] = sum;
    __syncthreads();

    if (first_row >= 0) {
        int t = tid - 1;
        while (t >= 0 && s_crow[t] == first_row) --t;
        double acc = 0.0;
        for (int u = t + 1; u < tid; ++u) acc += s_cval[u];
        acc += first_val;
        if (t < 0 && first_row == 0 && k0 > s_rowstart0) {
            a.head_row[tile] = r0;
            a.head_val[tile] = acc;
        } else {
            epi(r0 + first_row, acc);
        }
    }
    if (tid == kSpmvThreads - 1) {
        const int crow = s_crow[tid];
        if (r0 + crow < a.m) {
            int t = tid;
            while (t >= 0 && s_crow[t] == crow) --t;
            double acc = 0.0;
            for (int u = t + 1; u <= tid; ++u) acc += s_cval[u];
            a.carry_row[tile] = r0 + crow;
            a.carry_val[tile] = acc;
        } else {
            a.carry_row[tile] = -1;
        }
    }
}

// Finishes the row that began before `tile` and ends in it, if there is one:
// the carries of the tiles before it that hold nothing but that row, in order.
// kFixBatch loads at a time, past L1 (in one launch other SMs wrote them): one
// after the other a row over 1,675 tiles took 411 us, with L1 217.
constexpr int kFixBatch = 16;
template <class Epi>
__device__ __forceinline__ void fix_up(const SpmvMat& a, int64_t tile, const Epi& epi) {
    const int r = __ldcg(a.head_row + tile);
    if (r < 0) return;
    int64_t first = tile;
    for (int n = kFixBatch; n == kFixBatch; first -= n) {
        int row[kFixBatch];
#pragma unroll
        for (int u = 0; u < kFixBatch; ++u) row[u] = first - 1 - u >= 0 ? __ldcg(a.carry_row + first - 1 - u) : -1;
        n = 0;
#pragma unroll
        for (int u = 0; u < kFixBatch; ++u) n += n == u && row[u] == r;
    }
    double acc = 0.0;
    for (int64_t t = first; t < tile; t += kFixBatch) {
        double v[kFixBatch];
#pragma unroll
        for (int u = 0; u < kFixBatch; ++u) v[u] = t + u < tile ? __ldcg(a.carry_val + t + u) : 0.0;
#pragma unroll
        for (int u = 0; u < kFixBatch; ++u)
            if (t + u < tile) acc += v[u];
    }
    acc += __ldcg(a.head_val + tile);
    epi(r, acc);
}

template <class Epi>
__global__ void spmv_fixup_kernel(SpmvMat a, Epi epi) {
    if (!after_previous()) return;
    const int64_t tile = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (tile < a.ntiles) fix_up(a, tile, epi);
}

// ---- the merge path in one launch, for matrices of few tiles ----
// The same tiles, items and association as spmv_tile_kernel + fix-up, bit for
// bit; what differs is latency, which is all that a small product costs. The
// tile's nonzeros are read in order (coalesced, as soon as its corner is
// known) and multiplied into shared memory while the row ends arrive and the
// threads search the path, instead of after the search. A row that began in
// an earlier tile needs that tile's carry: where no row has more than kHeadNnz
// entries before a tile's start (short_heads, found with the tile table) the
// tile forms the carry itself, from the same products in the same groups of
// kSpmvIpt items; otherwise the last tile to finish does the fix-ups, 2 us
// more. Two products can share a launch.
// y = A x - b and A^T lam of 200 x 500: 10.0 us of kernels in two launches, 17.5
// in four (24.6 -> 12.3 us a pair of calls, 9.5 with launches prepared ahead);
// the one iteration's products of 2,000 x 5,000: 6 us each instead of 9.5.
// Where it stops paying, us in one launch and in two. Short heads, rows of 8 and
// of 40 entries: 600 tiles 9.9 and 13.8, 12.2 and 16.0; 1,184 tiles 16.0 and
// 17.0, 18.5 and 18.8; 2,000 tiles 23.5 and 24.9, 26.7 and 26.5; 3,000 tiles
// 33.4 and 32.9, 37.1 and 35.3. With the ticket, where one CTA walks all heads,
// rows of 2,000 and of 100,000 entries: 296 tiles 19.6 and 18.7, 18.0 and 18.9;
// 444 tiles 19.9 and 20.0, 18.2 and 20.3; 600 tiles 23.2 and 22.8, 22.7 and
// 21.7; 1,000 tiles 32.8 and 25.4, 37.3 and 25.5.
constexpr int64_t kSpmvSmallTiles = 2048, kSpmvTicketTiles = 444;
struct SmallTile {
    double prod[kSpmvTile];
    int32_t rowend[kSpmvTile + 1];
    int32_t crow[kSpmvThreads];
    double cval[kSpmvThreads];
    double head[kHeadNnz];
    double carry;
    bool last;
};

// kTicket: the fix-ups are the last tile's. A form of its own, or the other one
// has its registers too (64 instead of 40 or 48: 11.8 us instead of 9.9 at 600 tiles).
template <bool kTicket, class Epi>
__device__ __forceinline__ void small_tile(const SpmvMat& a, const double* __restrict__ x, const Epi& epi, int tile,
                                           SmallTile& sh) {
    const int tid = threadIdx.x;
    const int r0 = a.tile_row[tile], k0 = a.tile_nz[tile];
    const int nrows_t = a.tile_row[tile + 1] - r0, nnz_t = a.tile_nz[tile + 1] - k0;
    {
        int c[kSpmvIpt];
        double w[kSpmvIpt];
#pragma unroll
        for (int u = 0; u < kSpmvIpt; ++u) {
            const int i = tid + u * kSpmvThreads;
            c[u] = i < nnz_t ? __ldg(a.ci + k0 + i) : 0;
            w[u] = i < nnz_t ? __ldg(a.val + k0 + i) : 0.0;
        }
#pragma unroll
        for (int u = 0; u <= kSpmvIpt; ++u) {
            const int i = tid + u * kSpmvThreads;
            if (i <= nrows_t) sh.rowend[i] = r0 + i < a.m ? __ldg(a.rp + r0 + i + 1) : INT_MAX;
        }
#pragma unroll
        for (int u = 0; u < kSpmvIpt; ++u) {
            const int i = tid + u * kSpmvThreads;
            if (i < nnz_t) sh.prod[i] = w[u] * __ldcg(x + c[u]);
        }
    }
    const int rowstart0 = r0 < a.m ? __ldg(a.rp + r0) : a.nnz;
    if constexpr (kTicket) {
        if (tid == 0) a.head_row[tile] = -1;
    } else if (tid >= kSpmvThreads - 32 && k0 > rowstart0 && nrows_t > 0) {
        // the last warp: the carry of the row that ends here and began in the tile before
        const int n = k0 - rowstart0, lane = tid & 31;
        const int off = r0 - a.tile_row[tile - 1] + rowstart0 - a.tile_nz[tile - 1];  // item of its first entry
        for (int i = lane; i < n; i += 32) sh.head[i] = __ldg(a.val + rowstart0 + i) * __ldcg(x + __ldg(a.ci + rowstart0 + i));
        __syncwarp();
        if (lane == 0) {
            double acc = 0.0, part = 0.0;
            for (int i = 0; i < n; ++i) {
                part += sh.head[i];
                if ((off + i + 1) % kSpmvIpt == 0) {  // the last of its thread's items
                    acc += part;
                    part = 0.0;
                }
            }
            if ((off + n) % kSpmvIpt != 0) acc += part;
            sh.carry = acc;
        }
    }
    __syncthreads();

    const int total_t = nrows_t + nnz_t;
    const int diag = min(tid * kSpmvIpt, total_t);
    const int diag_end = min(diag + kSpmvIpt, total_t);
    int row = tile_search(sh.rowend, k0, diag, nrows_t, nnz_t);
    int nz = diag - row;
    double sum = 0.0;
    int first_row = -1;
    double first_val = 0.0;
#pragma unroll
    for (int it = 0; it < kSpmvIpt; ++it) {
        if (diag + it < diag_end) {
            if (nz < nnz_t && k0 + nz < sh.rowend[row]) {
                sum += sh.prod[nz];
                ++nz;
            } else if (row < nrows_t) {
                if (first_row < 0) {
                    first_row = row;
                    first_val = sum;
                } else {
                    epi(r0 + row, sum);
                }
                sum = 0.0;
                ++row;
            }
        }
    }
    sh.crow[tid] = row;
    sh.cval[tid] = sum;
    __syncthreads();
    if (first_row >= 0) {
        int t = tid - 1;
        while (t >= 0 && sh.crow[t] == first_row) --t;
        double acc = 0.0;
        for (int u = t + 1; u < tid; ++u) acc += sh.cval[u];
        acc += first_val;
        const bool head = t < 0 && first_row == 0 && k0 > rowstart0;
        if (kTicket && head) {
            a.head_row[tile] = r0;
            a.head_val[tile] = acc;
        } else {
            epi(r0 + first_row, head ? (0.0 + sh.carry) + acc : acc);
        }
    }
    if constexpr (!kTicket) return;
    if (tid == kSpmvThreads - 1) {
        const int crow = sh.crow[tid];
        if (r0 + crow < a.m) {
            int t = tid;
            while (t >= 0 && sh.crow[t] == crow) --t;
            double acc = 0.0;
            for (int u = t + 1; u <= tid; ++u) acc += sh.cval[u];
            a.carry_row[tile] = r0 + crow;
            a.carry_val[tile] = acc;
        } else {
            a.carry_row[tile] = -1;
        }
    }
    __threadfence();
    __syncthreads();
    // the count wraps to zero by itself: a reset of its own would lose the counts of
    // a product that overlaps this one (against the rules), and with them every later fix-up
    if (tid == 0) sh.last = atomicInc(a.ticket, (unsigned)(a.ntiles - 1)) == (unsigned)(a.ntiles - 1);
    __syncthreads();
    if (!sh.last) return;
    __threadfence();
    for (int64_t t = tid; t < a.ntiles; t += kSpmvThreads) fix_up(a, t, epi);
}

template <bool kTicket, class Epi>
__global__ void __launch_bounds__(kSpmvThreads) spmv_small_kernel(SpmvMat a, const double* __restrict__ x, Epi epi) {
    if (!after_previous()) return;
    __shared__ SmallTile sh;
    small_tile<kTicket>(a, x, epi, blockIdx.x, sh);
}

template <bool kTicket, bool kTicket2, class Epi, class Epi2>
__global__ void __launch_bounds__(kSpmvThreads) spmv_small2_kernel(SpmvMat a, const double* __restrict__ x, Epi epi,
                                                                   SpmvMat b, const double* __restrict__ x2,
                                                                   Epi2 epi2) {
    if (!after_previous()) return;
    __shared__ SmallTile sh;
    if (blockIdx.x < (unsigned)a.ntiles)
        small_tile<kTicket>(a, x, epi, blockIdx.x, sh);
    else
        small_tile<kTicket2>(b, x2, epi2, blockIdx.x - (int)a.ntiles, sh);
}

inline bool spmv_ticket(const SpmvMat& M) { return M.ntiles > 1 && !M.short_heads; }
inline bool spmv_small(const SpmvMat& M) {
    return M.kind == 0 && M.ticket && M.ntiles <= (spmv_ticket(M) ? kSpmvTicketTiles : kSpmvSmallTiles);
}

// ---- binned vector CSR ----
// A group of G lanes sums one row: lane l takes the row's nonzeros l, l + G,
// ... in order (kVecUnroll loads in flight), then the group combines its
// lanes by a fixed shuffle tree; every row's association order is fixed, so
// results are deterministic. Rows are grouped by G (bins); one launch covers
// all bins.
constexpr int kVecUnroll = 4;

template <int G, class Epi>
__device__ __forceinline__ void vec_rows(const SpmvMat& a, int bin, int unit, const double* __restrict__ x,
                                         const Epi& epi) {
    const int lane = threadIdx.x & 31, sub = lane / G, l = lane % G;
    const int idx = a.bins.row_off[bin] + unit * (32 / G) + sub;
    const bool valid = idx < a.bins.row_off[bin + 1];
    const int r = valid ? a.perm[idx] : 0;
    const int k0 = valid ? __ldg(a.rp + r) : 0, k1 = valid ? __ldg(a.rp + r + 1) : 0;
    double sum = 0.0;
    for (int k = k0 + l; k < k1; k += kVecUnroll * G) {
        int c[kVecUnroll];
        double w[kVecUnroll];
#pragma unroll
        for (int u = 0; u < kVecUnroll; ++u) {
            const int kk = k + u * G;
            c[u] = kk < k1 ? __ldg(a.ci + kk) : 0;
            w[u] = kk < k1 ? __ldg(a.val + kk) : 0.0;
        }
        double p[kVecUnroll];
#pragma unroll
        for (int u = 0; u < kVecUnroll; ++u) p[u] = (k + u * G < k1) ? w[u] * __ldcg(x + c[u]) : 0.0;
#pragma unroll
        for (int u = 0; u < kVecUnroll; ++u)
            if (k + u * G < k1) sum += p[u];
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o, G);
    if (valid && l == 0) epi(r, sum);
}

template <class Epi>
__global__ void __launch_bounds__(kSpmvThreads) spmv_vec_kernel(SpmvMat a, const double* __restrict__ x, Epi epi) {
    if (!after_previous()) return;
    const int w = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    if (w >= a.bins.unit_off[a.bins.nbins]) return;  // whole warps leave together
    int bin = 0;
    while (w >= a.bins.unit_off[bin + 1]) ++bin;
    const int unit = w - a.bins.unit_off[bin];
    switch (a.bins.lg[bin]) {
        case 0: vec_rows<1>(a, bin, unit, x, epi); break;
        case 1: vec_rows<2>(a, bin, unit, x, epi); break;
        case 2: vec_rows<4>(a, bin, unit, x, epi); break;
        case 3: vec_rows<8>(a, bin, unit, x, epi); break;
        case 4: vec_rows<16>(a, bin, unit, x, epi); break;
        default: vec_rows<32>(a, bin, unit, x, epi); break;
    }
}

// Launches one product on `s`: the binned vector kernel, or the merge-path
// tile kernel and its fix-up.
template <class Epi>
void spmv_launch(const SpmvMat& M, const double* x, const Epi& epi, cudaStream_t s) {
    if (M.kind == 1) {
        const int64_t units = M.bins.unit_off[M.bins.nbins];
        if (units == 0) return;
        launch_next(spmv_vec_kernel<Epi>, (unsigned)((units * 32 + kSpmvThreads - 1) / kSpmvThreads), kSpmvThreads, 0,
                    s, M, x, epi);
        launched("spmv_vec_kernel");
        return;
    }
    if (M.ntiles == 0) return;
    if (spmv_small(M)) {
        launch_next(spmv_ticket(M) ? spmv_small_kernel<true, Epi> : spmv_small_kernel<false, Epi>, (unsigned)M.ntiles,
                    kSpmvThreads, 0, s, M, x, epi);
        launched("spmv_small_kernel");
        return;
    }
    launch_next(spmv_tile_kernel<Epi>, (unsigned)M.ntiles, kSpmvThreads, 0, s, M, x, epi);
    launched("spmv_tile_kernel");
    if (M.ntiles > 1) {
        launch_next(spmv_fixup_kernel<Epi>, (unsigned)((M.ntiles + 255) / 256), 256, 0, s, M, epi);
        launched("spmv_fixup_kernel");
    }
}

// Two products that do not depend on one another, in one launch where both are small.
template <class Epi, class Epi2>
void spmv_launch2(const SpmvMat& M, const double* x, const Epi& epi, const SpmvMat& M2, const double* x2,
                  const Epi2& epi2, cudaStream_t s) {
    if (spmv_small(M) && spmv_small(M2) && M.ntiles > 0 && M2.ntiles > 0) {
        auto* kernel = spmv_ticket(M) ? (spmv_ticket(M2) ? spmv_small2_kernel<true, true, Epi, Epi2>
                                                         : spmv_small2_kernel<true, false, Epi, Epi2>)
                                      : (spmv_ticket(M2) ? spmv_small2_kernel<false, true, Epi, Epi2>
                                                         : spmv_small2_kernel<false, false, Epi, Epi2>);
        launch_next(kernel, (unsigned)(M.ntiles + M2.ntiles), kSpmvThreads, 0, s, M, x, epi, M2, x2, epi2);
        launched("spmv_small2_kernel");
        return;
    }
    spmv_launch(M, x, epi, s);
    spmv_launch(M2, x2, epi2, s);
}

// ---- epilogues ----
struct EpiAxpby {
    double alpha, beta;
    double* y;
    __device__ __forceinline__ void operator()(int r, double s) const {
        y[r] = (beta == 0.0) ? alpha * s : alpha * s + beta * y[r];
    }
};

// y = s - b (a residual op(A) x - b in one pass)
struct EpiSub {
    const double* b;
    double* y;
    __device__ __forceinline__ void operator()(int r, double s) const { y[r] = s - b[r]; }
};

// IPM epilogues (core/lp/interior_point.cpp line numbers in hn_ipm.cu)
struct EpiResidual {
    const double* b;
    double* mx;
    double* rp;
    __device__ __forceinline__ void operator()(int r, double s) const {
        mx[r] = s;
        rp[r] = s - b[r];
    }
};

struct EpiDualResidual {
    const double* z;
    const double* c;
    double* rd;
    __device__ __forceinline__ void operator()(int j, double s) const { rd[j] = (s + z[j]) - c[j]; }
};

struct EpiRhs {
    const double* rp;
    const double* mx;
    double* rhs;
    __device__ __forceinline__ void operator()(int i, double s) const { rhs[i] = ((-rp[i]) - s) + mx[i]; }
};

struct EpiCorrRhs {
    const double* pred;
    double* rhs;
    __device__ __forceinline__ void operator()(int i, double s) const { rhs[i] = pred[i] - s; }
};

struct EpiDirection {
    const double* D;
    const double* rd;
    const double* x;
    const double* corr;
    double* dx;
    double* dz;
    __device__ __forceinline__ void operator()(int j, double s) const {
        const double u = s + rd[j];
        double v = D[j] * u - x[j];
        if (corr) v = v + corr[j];
        dx[j] = v;
        dz[j] = -u;
    }
};

}  // namespace hn
