// C ABI of the products: SpMV (A and A^T) and SpMM.
#include <cstring>

#include "hn_spmv.cuh"

namespace hn {
namespace {

// C = op(A) B, B row-major (ncols x k), nonzeros in CSR order so each C entry
// is summed in the reference's order (gpu_backend.cpp:112-121). Two kernels.
// More than 64 columns: one warp per row, lanes own output columns, kSpmmCols
// accumulators each.
constexpr int kSpmmCols = 4;  // 32 lanes x 4 = 128 columns per pass

__global__ void __launch_bounds__(256) spmm_wide_kernel(int m, const int32_t* __restrict__ rp,
                                                   const int32_t* __restrict__ ci,
                                                   const double* __restrict__ val,
                                                   const double* __restrict__ B, int64_t k,
                                                   double* __restrict__ C) {
    if (!after_previous()) return;
    const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= m) return;
    const int32_t p0 = rp[row], p1 = rp[row + 1];
    for (int64_t c0 = 0; c0 < k; c0 += 32 * kSpmmCols) {
        double acc[kSpmmCols];
#pragma unroll
        for (int u = 0; u < kSpmmCols; ++u) acc[u] = 0.0;
        for (int32_t p = p0; p < p1; ++p) {
            const double a = __ldg(val + p);
            const double* Bj = B + (int64_t)__ldg(ci + p) * k;
#pragma unroll
            for (int u = 0; u < kSpmmCols; ++u) {
                const int64_t c = c0 + u * 32 + lane;
                if (c < k) acc[u] += a * __ldg(Bj + c);
            }
        }
#pragma unroll
        for (int u = 0; u < kSpmmCols; ++u) {
            const int64_t c = c0 + u * 32 + lane;
            if (c < k) C[row * k + c] = acc[u];
        }
    }
}

// Up to 64 columns: G lanes per row, so that none is idle, CC columns each, and
// the indices and values of U nonzeros loaded together before their entries of
// B; with a warp per row, 20,000 x 50,000 with 8 per column took 22.7 us at any
// k up to 32, now 8.3 (k = 1, 3), 10.3 (8), 12.4 (16), 16.5 (32) and 22.6 (64;
// 26.8). The line, this form and the wide one: 20,000 x 50,000 with 20 per row
// 17.2 us and 19.3 at k = 64, 29.8 and 21.4 at 65 (another pass over the row),
// 34.0 and 30.6 at 128; 50,000 x 50,000 with 40 per row 75 and 84, 134 and 94,
// 149 and 131. Fewer lanes than columns (CC = 2 from 17 on) read B in fewer, longer lines; more nonzeros in
// flight than U only cost registers.
template <int G, int CC, int U>
__global__ void __launch_bounds__(256) spmm_kernel(int m, const int32_t* __restrict__ rp,
                                                   const int32_t* __restrict__ ci,
                                                   const double* __restrict__ val,
                                                   const double* __restrict__ B, int64_t k,
                                                   double* __restrict__ C) {
    if (!after_previous()) return;
    const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int l = threadIdx.x % G;
    if (row >= m) return;
    const int32_t p0 = __ldg(rp + row), p1 = __ldg(rp + row + 1);
    for (int64_t c0 = l; c0 < k; c0 += G * CC) {
        double acc[CC];
#pragma unroll
        for (int q = 0; q < CC; ++q) acc[q] = 0.0;
        for (int32_t p = p0; p < p1; p += U) {
            int32_t j[U];
            double a[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                j[u] = p + u < p1 ? __ldg(ci + p + u) : 0;
                a[u] = p + u < p1 ? __ldg(val + p + u) : 0.0;
            }
            double b[U][CC];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int q = 0; q < CC; ++q)
                    if (p + u < p1 && c0 + q * G < k) b[u][q] = __ldg(B + (int64_t)j[u] * k + c0 + q * G);
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int q = 0; q < CC; ++q)
                    if (p + u < p1 && c0 + q * G < k) acc[q] += a[u] * b[u][q];
        }
#pragma unroll
        for (int q = 0; q < CC; ++q)
            if (c0 + q * G < k) C[row * k + c0 + q * G] = acc[q];
    }
}

template <int G, int CC, int U>
void spmm_launch(const SpmvMat& M, const double* B, int64_t k, double* C, cudaStream_t s) {
    const int64_t threads = (int64_t)M.m * G;
    launch_next(spmm_kernel<G, CC, U>, (unsigned)((threads + 255) / 256), 256, 0, s, M.m, M.rp, M.ci, M.val, B, k, C);
    launched("spmm_kernel");
}

void check_handle(const hn_csr* A, int trans) {
    if (!A) fail(HN_ERR_INVALID_ARG, "null matrix handle");
    if (trans && !A->has_t) fail(HN_ERR_INVALID_ARG, "handle was created without A^T");
}

void spmm_run(const hn_csr* A, int trans, const double* B, int64_t k, double* C, cudaStream_t s) {
    const SpmvMat M = spmv_mat(A, trans);
    if (M.m == 0 || k == 0) return;
    if (k > 64) {
        launch_next(spmm_wide_kernel, (unsigned)(((int64_t)M.m * 32 + 255) / 256), 256, 0, s, M.m, M.rp, M.ci, M.val,
                    B, k, C);
        launched("spmm_wide_kernel");
    } else if (k > 32) {
        spmm_launch<32, 2, 1>(M, B, k, C, s);
    } else if (k > 16) {
        spmm_launch<16, 2, 2>(M, B, k, C, s);
    } else if (k > 8) {
        spmm_launch<16, 1, 4>(M, B, k, C, s);
    } else if (k > 4) {
        spmm_launch<8, 1, 4>(M, B, k, C, s);
    } else if (k > 2) {
        spmm_launch<4, 1, 4>(M, B, k, C, s);
    } else {
        spmm_launch<2, 1, 4>(M, B, k, C, s);
    }
}

}  // namespace
}  // namespace hn

using namespace hn;

extern "C" {

int hn_spmv(const hn_csr* A, int trans, double alpha, const double* x, double beta, double* y,
            void* stream) {
    return guard("hn_spmv", [&] {
        require_init();
        check_handle(A, trans);
        const SpmvMat M = spmv_mat(A, trans);
        const int64_t cols = trans ? A->m : A->n;
        if (M.m > 0 && !y) fail(HN_ERR_INVALID_ARG, "null y");
        if (cols > 0 && M.nnz > 0 && !x) fail(HN_ERR_INVALID_ARG, "null x");
        spmv_launch(M, x, EpiAxpby{alpha, beta, y}, as_stream(stream));
    });
}

int hn_spmv_residual(const hn_csr* A, int trans, const double* x, const double* b, double* y, void* stream) {
    return guard("hn_spmv_residual", [&] {
        require_init();
        check_handle(A, trans);
        const SpmvMat M = spmv_mat(A, trans);
        const int64_t cols = trans ? A->m : A->n;
        if (M.m > 0 && (!y || !b)) fail(HN_ERR_INVALID_ARG, "null b or y");
        if (cols > 0 && M.nnz > 0 && !x) fail(HN_ERR_INVALID_ARG, "null x");
        spmv_launch(M, x, EpiSub{b, y}, as_stream(stream));
    });
}

int hn_spmv_host(const hn_csr* A, int trans, const double* x, double* y) {
    return guard("hn_spmv_host", [&] {
        require_init();
        check_handle(A, trans);
        const SpmvMat M = spmv_mat(A, trans);
        const int64_t cols = trans ? A->m : A->n;
        const int64_t rows = M.m;
        if ((rows > 0 && !y) || (cols > 0 && !x)) fail(HN_ERR_INVALID_ARG, "null vector");
        cudaStream_t s = nullptr;
        Workspace& w = workspace(s);
        ensure_staging(w, sizeof(double) * (cols + rows + 2), s);
        double* xh = w.staging_h;
        double* yh = w.staging_h + cols;
        double* xd = w.staging_d;
        double* yd = w.staging_d + cols;
        std::memcpy(xh, x, sizeof(double) * cols);
        check_cuda(cudaMemcpyAsync(xd, xh, sizeof(double) * cols, cudaMemcpyHostToDevice, s), "H2D x");
        spmv_launch(M, xd, EpiAxpby{1.0, 0.0, yd}, s);
        check_cuda(cudaMemcpyAsync(yh, yd, sizeof(double) * rows, cudaMemcpyDeviceToHost, s), "D2H y");
        check_cuda(cudaStreamSynchronize(s), "hn_spmv_host sync");
        std::memcpy(y, yh, sizeof(double) * rows);
    });
}

int hn_spmm(const hn_csr* A, int trans, const double* B, int64_t k, double* C, void* stream) {
    return guard("hn_spmm", [&] {
        require_init();
        check_handle(A, trans);
        if (k < 0) fail(HN_ERR_INVALID_ARG, "negative k");
        spmm_run(A, trans, B, k, C, as_stream(stream));
    });
}

int hn_spmm_host(const hn_csr* A, int trans, const double* B, int64_t k, double* C) {
    return guard("hn_spmm_host", [&] {
        require_init();
        check_handle(A, trans);
        if (k < 0) fail(HN_ERR_INVALID_ARG, "negative k");
        const int64_t cols = trans ? A->m : A->n;
        const int64_t rows = trans ? A->n : A->m;
        cudaStream_t s = nullptr;
        Workspace& w = workspace(s);
        const size_t nb = sizeof(double) * (size_t)(cols * k), nc = sizeof(double) * (size_t)(rows * k);
        ensure_staging(w, nb + nc + 16, s);
        double* Bd = w.staging_d;
        double* Cd = w.staging_d + cols * k;
        std::memcpy(w.staging_h, B, nb);
        check_cuda(cudaMemcpyAsync(Bd, w.staging_h, nb, cudaMemcpyHostToDevice, s), "H2D B");
        spmm_run(A, trans, Bd, k, Cd, s);
        check_cuda(cudaMemcpyAsync(w.staging_h + cols * k, Cd, nc, cudaMemcpyDeviceToHost, s), "D2H C");
        check_cuda(cudaStreamSynchronize(s), "hn_spmm_host sync");
        std::memcpy(C, w.staging_h + cols * k, nc);
    });
}

}  // extern "C"
