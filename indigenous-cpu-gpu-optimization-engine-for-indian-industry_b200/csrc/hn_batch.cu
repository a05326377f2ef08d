// Batched Mehrotra IPM: many LPs of uneven sizes advanced in lockstep.
//
// The instances are packed as one block-diagonal CSR M = diag(M_1 .. M_K)
// (rows row_off[i]..row_off[i+1], columns col_off[i]..col_off[i+1]), so the
// merge-path SpMVs with their IPM epilogues, the device A^T and the A D A^T
// assembly run on the whole batch in single launches (the assembly's
// per-row windows keep its bitmaps to one block). What differs per instance
// lives here:
//   - reductions per instance (one CTA each): mu, ||rp||_inf, ||rd||_inf, step
//     lengths, mu_aff, sigma -- the scalars of interior_point.cpp:517-530,
//     :629-643, :683-684 -- in a K x HN_IPM_NSCAL block, plus a per-instance
//     status word (0 = iterating) that masks converged or failed instances out
//     of the factorisation, the solves and the update;
//   - dyn_reg = max(reg, 1e-12 * max diag) per instance (:188-196);
//   - the normal-equation factorisation: each instance's N block is scattered
//     into a dense lower triangle and factorised by a blocked LDL^T on the GPU
//     with the reference's pivot clamp (factorization.cpp:1299-1305), level-
//     synchronously in 64-column blocks: per block one launch factorises every
//     instance's diagonal block, one spreads all instances' panel rows and one
//     all instances' output tiles over the GPU. This is a deliberate
//     deviation from keeping factorisations on the host: thousands of
//     factorisations per iteration do not fit in host time;
//   - the two triangular solves, one launch for the batch (a CTA or a cluster
//     of CTAs per instance), and iterative refinement (refinement.cpp:7-37: up to 5 sweeps, stop at
//     1e-10 relative) per instance, with N x as one SpMV over the packed N.
#include <algorithm>
#include <cmath>
#include <numeric>
#include <type_traits>
#include <vector>

#include "hn_spmv.cuh"

namespace hn {
// Where an instance lies: one 32-byte load instead of a chain through the offsets.
struct __align__(16) InstInfo {
    int64_t r0;  // first packed row
    int64_t dn;  // offset of its dense block
    int32_t m;
    int32_t pad[3];
};

// A chunk of 256 (kT) rows below a diagonal block: its instance and its number there.
struct Chunk {
    int32_t inst, local;
};

// What a CTA of the solve kernel works on.
struct SolveSlot {
    int32_t inst;   // -1: nothing (its cluster's barriers only)
    int32_t rank, size;
    int32_t steps;  // blocks of the largest instance in the cluster, 0: its instances are all one CTA's
};

}  // namespace hn

struct hn_batch {
    int64_t K = 0, m = 0, n = 0;
    const hn_pattern* P = nullptr;
    int64_t* row_off = nullptr;  // K+1
    int64_t* col_off = nullptr;  // K+1
    int32_t* row_inst = nullptr; // m
    int64_t* dn_off = nullptr;   // K+1, offsets of the dense blocks
    int32_t* order = nullptr;    // instances by decreasing size
    double* dense = nullptr;     // sum m_i^2
    double* dD = nullptr;        // LDL^T pivots, m
    int32_t* refine = nullptr;   // per-instance refinement flag (1 = keep sweeping)
    int32_t* nref = nullptr;     // instances still refining, blocks that have counted; zero between launches
    int32_t* left_host = nullptr;  // the former, in pinned host memory
    // N as an SpMV operand (int32 row pointer copy + merge-path tables)
    int32_t* nrp = nullptr;
    int64_t ntiles = 0;
    int32_t *tile_row = nullptr, *tile_nz = nullptr, *carry_row = nullptr, *head_row = nullptr;
    double *carry_val = nullptr, *head_val = nullptr;
    bool short_heads = false;
    double* r = nullptr;         // refinement residual, m
    double* ax = nullptr;        // N x, m
    hn::InstInfo* info = nullptr;  // K
    // level schedule of the blocked factorisation: at block step s the
    // instances order[0 .. cnt[s]) still have a block. Their 64 x 64 output
    // tiles of the update that follows step s (the next block column after an
    // even step, the whole trailing triangle after an odd one) as cumulative
    // counts per (step, instance), and the kT-row chunks below their diagonal
    // blocks as a list per step, spread every instance's work over the GPU.
    int64_t mmax = 0, nsteps = 0;  // rows and blocks of the largest instance
    std::vector<int32_t> step_cnt;                       // host, nsteps
    std::vector<int64_t> tile_off_h, chunk_off_h;        // host, nsteps+1 offsets into the two tables
    std::vector<int64_t> step_tiles_h;                   // host, tiles per step
    int64_t* step_tiles = nullptr;                       // device
    hn::Chunk* chunks = nullptr;                         // device
    int64_t nslots = 0, solve_smem = 0;
    hn::SolveSlot* slots = nullptr;  // the solve kernel's CTAs, whole clusters
    double* work = nullptr;          // solved blocks of the forward pass, m
    double* solve_part = nullptr;    // backward partial dot products, two times 64 per chunk
    // relative KKT residual per instance and the tightening past the
    // reference's stop (hn_batch_set_kkt): ru / cu / offset are caller-owned
    // unscale factors (null = not measured); kkt and kkt_ref hold K x 4
    // (residual, primal, dual, gap) at the last residual call and at the
    // iteration the reference's rule first held (ref_iter, -1 = not yet);
    // xb / zb / lb keep the iterate of that iteration
    const double *ru = nullptr, *cu = nullptr, *offset = nullptr;
    double kkt_tol = 0.0;
    int kkt_extra = 0;
    double *kkt = nullptr, *kkt_ref = nullptr;
    int32_t* ref_iter = nullptr;
    double *xb = nullptr, *zb = nullptr, *lb = nullptr;
};

namespace hn {
namespace {

constexpr int kT = 256;
constexpr int S_NRP = HN_IPM_NRP, S_NRD = HN_IPM_NRD, S_MU = HN_IPM_MU, S_AP = HN_IPM_AP, S_AD = HN_IPM_AD,
              S_MUAFF = HN_IPM_MUAFF, S_SIGMA = HN_IPM_SIGMA;
constexpr int ST_RUN = 0, ST_OPTIMAL = 1, ST_NUMERICAL = 7;

// Row stride of an instance's dense block: m rounded up to even, so every row
// starts on a 16-byte boundary (16-byte asynchronous copies of the panels).
__host__ __device__ __forceinline__ int dense_ld(int m) { return (m + 1) & ~1; }

__device__ __forceinline__ bool fin(double v) { return isfinite(v); }

// ---- per-instance reductions ----
// What the residual pass needs for the relative KKT residual and the
// tightening: see hn_batch_set_kkt.
struct KktArgs {
    const double *lam, *b, *c, *ru, *cu, *offset;
    double *kkt, *kkt_ref, *xb, *zb, *lb;
    int32_t* ref_iter;
    double tol;
    int extra;
};

__device__ __forceinline__ double fin_or_inf(double t) { return t <= 1.7976931348623157e308 ? t : INFINITY; }

__global__ void __launch_bounds__(kT) batch_prep_kernel(const int64_t* __restrict__ row_off,
                                                        const int64_t* __restrict__ col_off,
                                                        const double* __restrict__ x, const double* __restrict__ z,
                                                        const double* __restrict__ rd, const double* __restrict__ rp,
                                                        double* __restrict__ D, double* __restrict__ Drd,
                                                        double* __restrict__ scal, int32_t* __restrict__ status,
                                                        int32_t* __restrict__ iters, int iter, double tol,
                                                        double ctol, KktArgs k) {
    if (!after_previous()) return;
    __shared__ double sh[32];
    __shared__ int s_save;
    const int64_t i = blockIdx.x;
    const int64_t c0 = col_off[i], c1 = col_off[i + 1], r0 = row_off[i], r1 = row_off[i + 1];
    const bool measure = k.ru != nullptr;
    double smu = 0.0, mrd = 0.0, mrp = 0.0, du = 0.0, cn = 0.0, cx = 0.0, pr = 0.0, bn = 0.0, by = 0.0;
    for (int64_t j = c0 + threadIdx.x; j < c1; j += kT) {
        const double xj = x[j], zj = z[j], r = rd[j];
        smu += xj * zj;
        mrd = fmax(mrd, fabs(r));
        double d = xj / zj;
        if (!(d >= 0.0) || !fin(d) || d > 1e10) d = 1e10;  // interior_point.cpp:532-539
        D[j] = d;
        Drd[j] = d * r;
        if (measure) {
            const double u = k.cu[j], cj = k.c[j];
            du = fmax(du, fin_or_inf(fabs(r) * u));
            cn = fmax(cn, fabs(cj) * u);
            cx += cj * xj;
        }
    }
    for (int64_t q = r0 + threadIdx.x; q < r1; q += kT) {
        const double r = rp[q];
        mrp = fmax(mrp, fabs(r));
        if (measure) {
            const double u = k.ru[q], bq = k.b[q];
            pr = fmax(pr, fin_or_inf(fabs(r) * u));
            bn = fmax(bn, fabs(bq) * u);
            by += bq * k.lam[q];
        }
    }
    smu = block_sum<kT>(smu, sh);
    mrd = block_max<kT>(mrd, sh);
    mrp = block_max<kT>(mrp, sh);
    if (measure) {
        du = block_max<kT>(du, sh);
        cn = block_max<kT>(cn, sh);
        cx = block_sum<kT>(cx, sh);
        pr = block_max<kT>(pr, sh);
        bn = block_max<kT>(bn, sh);
        by = block_sum<kT>(by, sh);
    }
    if (threadIdx.x == 0) {
        const double mu = smu / static_cast<double>(c1 - c0);
        double* s = scal + i * HN_IPM_NSCAL;
        s[S_MU] = mu;
        s[S_NRD] = mrd;
        s[S_NRP] = mrp;
        double kk = 0.0;
        if (measure) {
            const double P = pr / (1.0 + bn), Dl = du / (1.0 + cn),
                         Gp = fabs(cx - by) / (1.0 + fabs(cx + k.offset[i]));
            kk = (P != P || Dl != Dl || Gp != Gp) ? nan("") : fmax(P, fmax(Dl, Gp));
            double* o = k.kkt + 4 * i;
            o[0] = kk;
            o[1] = P;
            o[2] = Dl;
            o[3] = Gp;
        }
        int save = 0;
        if (status[i] == ST_RUN) {
            int r = k.ref_iter[i];
            if (r < 0 && mrp < tol && mrd < tol && mu < ctol) {  // the reference's rule, :525-530
                r = iter;
                k.ref_iter[i] = iter;
                save = measure && k.tol > 0.0;
                if (measure)
                    for (int q = 0; q < 4; ++q) k.kkt_ref[4 * i + q] = k.kkt[4 * i + q];
            }
            // stop at the reference's rule, or past it once the KKT residual
            // is within tolerance or the extra iterations are spent
            if (r >= 0 && (!(measure && k.tol > 0.0) || kk <= k.tol || iter - r >= k.extra)) {
                status[i] = ST_OPTIMAL;
                iters[i] = iter;
            }
        }
        s_save = save;
    }
    __syncthreads();
    if (s_save) {  // keep the iterate the reference would return
        for (int64_t j = c0 + threadIdx.x; j < c1; j += kT) {
            k.xb[j] = x[j];
            k.zb[j] = z[j];
        }
        for (int64_t q = r0 + threadIdx.x; q < r1; q += kT) k.lb[q] = k.lam[q];
    }
}

// After the last residual pass: an instance that met the reference's rule
// and then failed (status 7), was still iterating, or ended with a larger
// KKT residual than at that point gets the saved iterate back.
__global__ void __launch_bounds__(kT) batch_finish_kernel(const int64_t* __restrict__ row_off,
                                                          const int64_t* __restrict__ col_off, double* __restrict__ x,
                                                          double* __restrict__ z, double* __restrict__ lam,
                                                          int32_t* __restrict__ status, int32_t* __restrict__ iters,
                                                          KktArgs k) {
    if (!after_previous()) return;
    __shared__ int s_restore;
    const int64_t i = blockIdx.x;
    const int r = k.ref_iter[i];
    if (r < 0) return;
    if (threadIdx.x == 0) {
        const double now = k.kkt[4 * i], then = k.kkt_ref[4 * i];
        const int st = status[i];
        const bool worse = !(now <= then);  // NaN now counts as worse
        s_restore = (st == ST_NUMERICAL || worse) ? 1 : 0;
        status[i] = ST_OPTIMAL;
        if (s_restore) {
            iters[i] = r;
            for (int q = 0; q < 4; ++q) k.kkt[4 * i + q] = k.kkt_ref[4 * i + q];
        }
    }
    __syncthreads();
    if (!s_restore) return;
    const int64_t c0 = col_off[i], c1 = col_off[i + 1], r0 = row_off[i], r1 = row_off[i + 1];
    for (int64_t j = c0 + threadIdx.x; j < c1; j += kT) {
        x[j] = k.xb[j];
        z[j] = k.zb[j];
    }
    for (int64_t q = r0 + threadIdx.x; q < r1; q += kT) lam[q] = k.lb[q];
}

__global__ void __launch_bounds__(kT) batch_steps_kernel(const int64_t* __restrict__ row_off,
                                                         const int64_t* __restrict__ col_off,
                                                         const double* __restrict__ x, const double* __restrict__ dx,
                                                         const double* __restrict__ z, const double* __restrict__ dz,
                                                         const double* __restrict__ dlam, double* __restrict__ scal,
                                                         int32_t* __restrict__ status) {
    if (!after_previous()) return;
    __shared__ double sh[32];
    __shared__ int s_bad;
    const int64_t i = blockIdx.x;
    if (status[i] != ST_RUN) return;
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
    const int64_t c0 = col_off[i], c1 = col_off[i + 1], r0 = row_off[i], r1 = row_off[i + 1];
    double ap = 1.0, ad = 1.0;
    bool bad = false;
    for (int64_t j = c0 + threadIdx.x; j < c1; j += kT) {
        const double a = dx[j], b = dz[j];
        if (a < 0.0) ap = fmin(ap, -x[j] / a);
        if (b < 0.0) ad = fmin(ad, -z[j] / b);
        bad |= !fin(a) || !fin(b);
    }
    for (int64_t k = r0 + threadIdx.x; k < r1; k += kT) bad |= !fin(dlam[k]);
    if (bad) s_bad = 1;
    ap = block_min<kT>(ap, sh);
    ad = block_min<kT>(ad, sh);
    if (threadIdx.x == 0) {
        double* s = scal + i * HN_IPM_NSCAL;
        const double sp = 0.99 * ap, sq = 0.99 * ad;  // max_step, :134-142
        s[S_AP] = sp < 1.0 ? sp : 1.0;
        s[S_AD] = sq < 1.0 ? sq : 1.0;
        if (s_bad) status[i] = ST_NUMERICAL;  // :617-627, :676-686
    }
}

// mu_aff, sigma and zs = (sigma mu - dx dz) (1/z) of one instance per CTA.
__global__ void __launch_bounds__(kT) batch_corr_kernel(const int64_t* __restrict__ col_off,
                                                        const double* __restrict__ x, const double* __restrict__ dx,
                                                        const double* __restrict__ z, const double* __restrict__ dz,
                                                        double* __restrict__ scal, const int32_t* __restrict__ status,
                                                        double* __restrict__ zs) {
    if (!after_previous()) return;
    __shared__ double sh[32];
    __shared__ double s_sm;
    const int64_t i = blockIdx.x;
    const int64_t c0 = col_off[i], c1 = col_off[i + 1];
    double* s = scal + i * HN_IPM_NSCAL;
    if (status[i] != ST_RUN) {
        for (int64_t j = c0 + threadIdx.x; j < c1; j += kT) zs[j] = 0.0;
        return;
    }
    const double ap = s[S_AP], ad = s[S_AD];
    double acc = 0.0;
    for (int64_t j = c0 + threadIdx.x; j < c1; j += kT) acc += (x[j] + ap * dx[j]) * (z[j] + ad * dz[j]);
    acc = block_sum<kT>(acc, sh);
    if (threadIdx.x == 0) {
        const double mu_aff = acc / static_cast<double>(c1 - c0);  // :632-636
        const double mu = s[S_MU];
        double sigma;
        if (!fin(mu_aff) || mu_aff < 0.0 || !(mu > 0.0)) {
            sigma = 0.5;
        } else {
            const double r = pow(mu_aff / fmax(mu, 1e-300), 3.0);
            sigma = r < 0.1 ? 0.1 : (r > 0.9 ? 0.9 : r);  // :638-643
        }
        s[S_MUAFF] = mu_aff;
        s[S_SIGMA] = sigma;
        s_sm = sigma * mu;
    }
    __syncthreads();
    const double sm = s_sm;
    for (int64_t j = c0 + threadIdx.x; j < c1; j += kT) {
        const double zinv = 1.0 / z[j];
        zs[j] = (sm - dx[j] * dz[j]) * zinv;  // :645-651
    }
}

__global__ void __launch_bounds__(kT) batch_update_kernel(const int64_t* __restrict__ row_off,
                                                          const int64_t* __restrict__ col_off, double* __restrict__ x,
                                                          const double* __restrict__ dx, double* __restrict__ z,
                                                          const double* __restrict__ dz, double* __restrict__ lam,
                                                          const double* __restrict__ dlam,
                                                          const double* __restrict__ scal,
                                                          int32_t* __restrict__ status, int32_t* __restrict__ iters,
                                                          int iter) {
    if (!after_previous()) return;
    __shared__ int s_bad;
    const int64_t i = blockIdx.x;
    if (status[i] != ST_RUN) return;
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
    const int64_t c0 = col_off[i], c1 = col_off[i + 1], r0 = row_off[i], r1 = row_off[i + 1];
    const double ap = scal[i * HN_IPM_NSCAL + S_AP], ad = scal[i * HN_IPM_NSCAL + S_AD];
    bool bad = false;
    for (int64_t j = c0 + threadIdx.x; j < c1; j += kT) {
        const double xn = x[j] + ap * dx[j];
        const double zn = z[j] + ad * dz[j];
        x[j] = xn;
        z[j] = zn;
        bad |= xn < 0.0 || zn < 0.0 || !fin(xn) || !fin(zn);  // :698-708
    }
    for (int64_t k = r0 + threadIdx.x; k < r1; k += kT) lam[k] += ad * dlam[k];
    if (bad) s_bad = 1;
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_bad)
            status[i] = ST_NUMERICAL;
        else
            iters[i] = iter + 1;
    }
}

// ---- normal equations per instance ----
__global__ void __launch_bounds__(kT) batch_reg_kernel(const int64_t* __restrict__ row_off,
                                                       const int64_t* __restrict__ diag_pos, double reg,
                                                       const int32_t* __restrict__ status, double* __restrict__ nval) {
    if (!after_previous()) return;
    __shared__ double sh[32];
    __shared__ double s_dyn;
    const int64_t i = blockIdx.x;
    if (status[i] != ST_RUN) return;
    const int64_t r0 = row_off[i], r1 = row_off[i + 1];
    double md = 0.0;
    for (int64_t r = r0 + threadIdx.x; r < r1; r += kT) md = fmax(md, nval[diag_pos[r]]);  // NaN ignored
    md = block_max<kT>(md, sh);
    if (threadIdx.x == 0) {
        const double dyn = 1e-12 * md;
        s_dyn = (reg < dyn) ? dyn : reg;  // std::max(regularization, 1e-12 * max_diag)
    }
    __syncthreads();
    const double dyn = s_dyn;
    for (int64_t r = r0 + threadIdx.x; r < r1; r += kT) nval[diag_pos[r]] += dyn;
}

// One warp per packed row: zero the dense lower row, then scatter N's entries.
__global__ void batch_dense_kernel(int64_t m, const int64_t* __restrict__ row_off, const int32_t* __restrict__ row_inst,
                                   const int64_t* __restrict__ dn_off, const int32_t* __restrict__ status,
                                   const int64_t* __restrict__ rpN, const int32_t* __restrict__ ciN,
                                   const double* __restrict__ nval, double* __restrict__ dense) {
    if (!after_previous()) return;
    const int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= m) return;
    const int inst = row_inst[r];
    if (status[inst] != ST_RUN) return;
    const int64_t b0 = row_off[inst], mi = row_off[inst + 1] - b0, lr = r - b0;
    double* row = dense + dn_off[inst] + lr * dense_ld(static_cast<int>(mi));
    for (int64_t c = lane; c <= lr; c += 32) row[c] = 0.0;
    __syncwarp();
    for (int64_t p = rpN[r] + lane; p < rpN[r + 1]; p += 32) {
        const int64_t c = (int64_t)ciN[p] - b0;
        if (c >= 0 && c <= lr) row[c] = nval[p];
    }
}

// Blocked LDL^T, level-synchronous over the batch, in blocks of kFb columns:
// block step s runs for every instance that still has a block s --
//   batch_ldlt_diag_kernel: one CTA per instance factorises the kFb x kFb
//     diagonal block (pivot clamp of factorization.cpp:1299-1305);
//   batch_ldlt_panel_kernel: every instance's panel below its diagonal block,
//     in chunks of kT rows spread over the GPU, one row per thread;
//   batch_ldlt_update_kernel: A_rc -= sum_q (L_rq D_q) L_cq on the FP64 tensor
//     cores (mma.sync m8n8k4, FP64 in and out), after an even step for the
//     next block column only, after an odd one for the rest of the trailing
//     matrix by both panels.
constexpr int kFb = 64;

// D(8x8) += A(8x4) B(4x8) in FP64 on the tensor cores. Fragments: lane l
// holds A[l/4][l%4], B[l%4][l/4] and D[l/4][2(l%4)], D[l/4][2(l%4)+1].
__device__ __forceinline__ void dmma_m8n8k4(double* d, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// Quotients by a common divisor, correctly rounded as a / d is, from its
// correctly rounded reciprocal y: two residual corrections q + (a - d q) y
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34(1), 1990: a quotient within one ulp, its
// exact residual and a correctly rounded reciprocal give the rounded
// quotient; the first step brings a y within one ulp). Independent quotients
// overlap, which divisions -- each a branch around its rare cases -- do not:
// 43 cycles of latency against 127 each. Holds while nothing under- or
// overflows on the way: in_range(a) or a zero, and good_divisor(d); a / d
// otherwise. The residual is formed as d q - a and subtracted: a zero keeps
// its sign that way (a - d q is +0 for a = -0, and -0 + 0 = +0).
__device__ __forceinline__ double quotient(double a, double d, double y) {
    double q = a * y;
    q = __fma_rn(-__fma_rn(d, q, -a), y, q);
    return __fma_rn(-__fma_rn(d, q, -a), y, q);
}
// 2^-400 <= |v| < 2^401: exponent field 623 .. 1423
__device__ __forceinline__ bool in_range(double v) {
    return ((static_cast<unsigned>(__double2hiint(v)) >> 20) & 0x7ffu) - 623u <= 800u;
}

// A divisor whose reciprocal() is the rounded one (the last Newton step may
// miss it for a mantissa of all ones) and positive, as quotient()'s zeros want it.
__device__ __forceinline__ bool good_divisor(double d) {
    const bool ones = static_cast<unsigned>(__double2loint(d)) == 0xffffffffu &&
                      (static_cast<unsigned>(__double2hiint(d)) & 0xfffffu) == 0xfffffu;
    return (static_cast<unsigned>(__double2hiint(d)) >> 20) - 623u <= 800u && !ones;  // in_range, sign bit clear
}

// 1 / d, correctly rounded, for good_divisor(d): Newton steps from the hardware's
// approximation, the last one from an iterate within one ulp (Markstein, as
// above); no branch.
__device__ __forceinline__ double reciprocal(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
#pragma unroll
    for (int i = 0; i < 2; ++i) y = __fma_rn(__fma_rn(-d, y, 1.0), y, y);
    return __fma_rn(__fma_rn(-d, y, 1.0), y, y);
}

__device__ __forceinline__ double divisor_reciprocal(double d) { return good_divisor(d) ? reciprocal(d) : 0.0; }

// As the panels divide (there it is written out: in a function of its own
// their kernel takes 61 us instead of 56).
__global__ void quotients_kernel(int64_t n, const double* __restrict__ a, const double* __restrict__ d,
                                 double* __restrict__ q) {
    if (!after_previous()) return;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = a[i], y = divisor_reciprocal(d[i]);
    q[i] = y == 0.0 || !(in_range(v) || v == 0.0) ? v / d[i] : quotient(v, d[i], y);
}

// LDL^T of one instance's diagonal block per CTA: a chain of 64 pivots (form
// the clamped pivot, divide its column, update), so its time is the latency
// of a pivot. Four pivots go per round, to share the exchange between the
// warps. Thread (r, g) keeps of row r the column quads 4 i + g (i = 0 .. 3) in
// registers. The threads that own quad 4 i + g read its 4 x 4 pivot block
// from shared memory, factorise it (all of them the same) and divide their
// row's four columns; a barrier later the owners of the next quad bring it up
// to date and publish its pivot block; the other columns are updated while
// the next round's divisions are under way. A barrier per pivot, its shuffle
// and its trip through shared memory cost more than the division. An element
// takes A_rc -= (l_rj d_j) l_cj for j ascending, each product and difference
// rounded, the reference's elimination order; what a thread computes above
// the diagonal or past the block is never read.
// 384 LPs of m 50-2000 (31 blocks): 585 us, 1,558 with the block in shared
// memory and two barriers per pivot; one wave of blocks 15 us (41 before).
// R: the rows that a CTA has threads for, 16, 32, 48 or 64, so that the step's
// largest block fits: many small instances are bound by how many CTAs an SM
// holds. The factorisation of 16,000 instances of 10 rows takes 288 us, of 32
// rows 914, of 48 rows 1,838 (with 64 rows in every case 668, 1,315 and 1,898;
// 448, 1,441 and 2,395 with the block in shared memory).
template <int R>
struct DiagShared {
    double A[R][R + 1];
    double lc[2][4][R];  // the round's four columns of L, by the parity of the round
    double pb[4][4];     // the next pivot block (its lower triangle)
    double d[R];
};

// a[4] -= a round's four columns: row factors w[q] = l_rq d_q, columns c .. c + 3
template <int R>
__device__ __forceinline__ void diag_update(double* a, const double* w, const double (*lc)[R], int c) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[e] -= w[q] * lc[q][c + e];
}

// Four pivots: the pivot block pb (lower triangle) gives d[q] and, in a, row
// r's four columns of L. `plain` divides; the other way is the fast one and
// returns false where its quotients may not be the rounded ones.
template <bool plain>
__device__ __forceinline__ bool diag_pivots(const double (*pb)[4], double tol, double* a, double* d) {
    double l[4][4], t[4][4];
    bool fine = true;
    auto ok = [](double v) { return in_range(v) || v == 0.0; };
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = q; e < 4; ++e) t[e][q] = pb[e][q];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        d[q] = t[q][q];
        if (d[q] <= tol) d[q] = tol;  // SparseCholesky pivot clamp
        const double y = plain ? 0.0 : reciprocal(d[q]);
        if (!plain) fine = fine && good_divisor(d[q]) && ok(a[q]);
#pragma unroll
        for (int e = q + 1; e < 4; ++e) {
            l[e][q] = plain ? t[e][q] / d[q] : quotient(t[e][q], d[q], y);
            if (!plain) fine = fine && ok(t[e][q]);
        }
        a[q] = plain ? a[q] / d[q] : quotient(a[q], d[q], y);
        const double wr = a[q] * d[q];
#pragma unroll
        for (int e = q + 1; e < 4; ++e) {
            const double we = l[e][q] * d[q];
#pragma unroll
            for (int f = q + 1; f <= e; ++f) t[e][f] -= we * l[f][q];
            a[e] -= wr * l[e][q];
        }
    }
    return fine;
}
__device__ __noinline__ void diag_pivots_plain(const double (*pb)[4], double tol, double* a, double* d) {
    diag_pivots<true>(pb, tol, a, d);
}

// Rounds 4 I .. 4 I + 3 (pivots 16 I .. 16 I + 15). On entry and return the
// columns right of the previous round's successor still lack that round (row
// factors w, columns of L of the parity before): each round's owners take it
// after their pivots, the others before the round's first barrier.
template <int I, int R>
__device__ __forceinline__ void diag_rounds(DiagShared<R>& sh, double (*a)[4], double* w, int nb, double tol, int r,
                                            int g) {
    constexpr int kNext = 16 * (I + 1) < R ? I + 1 : I;  // the quads after these rounds' (or none)
#pragma unroll 1
    for (int og = 0; og < 4; ++og) {
        const int j0 = 16 * I + 4 * og;
        if (j0 >= nb) return;
        double(*lc)[R] = sh.lc[og & 1];
        // the previous round's update right of this round's quad
        auto rest = [&]() {
            if (I == 0 && og == 0) return;
            const double(*lp)[R] = sh.lc[(og & 1) ^ 1];
            if (g > og) diag_update(a[I], w, lp, 16 * I + 4 * g);
#pragma unroll
            for (int i = I + 1; i < R / 16; ++i) diag_update(a[i], w, lp, 16 * i + 4 * g);
        };
        if (g == og) {
            double d[4], t[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) t[q] = a[I][q];
            if (!diag_pivots<false>(sh.pb, tol, a[I], d)) {
                diag_pivots_plain(sh.pb, tol, t, d);
#pragma unroll
                for (int q = 0; q < 4; ++q) a[I][q] = t[q];
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                lc[q][r] = a[I][q];
                sh.A[r][j0 + q] = a[I][q];
                if (r == 0) sh.d[j0 + q] = d[q];
            }
        } else {
            rest();
        }
        __syncthreads();
        if (g == og) rest();
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = lc[q][r] * sh.d[j0 + q];
        if (g == ((og + 1) & 3) && j0 + 4 < R) {  // the next round's owners
            if (og < 3)
                diag_update(a[I], w, lc, j0 + 4);
            else
                diag_update(a[kNext], w, lc, j0 + 4);
            if (r >= j0 + 4 && r < j0 + 8) {
#pragma unroll
                for (int e = 0; e < 4; ++e) sh.pb[r - j0 - 4][e] = og < 3 ? a[I][e] : a[kNext][e];
            }
        }
        __syncthreads();
    }
}

template <int R>
__global__ void __launch_bounds__(4 * R) batch_ldlt_diag_kernel(int s, const InstInfo* __restrict__ info,
                                                                const int32_t* __restrict__ order,
                                                                const int32_t* __restrict__ status,
                                                                double* __restrict__ dense, double* __restrict__ dD,
                                                                double tol) {
    const int inst = order[blockIdx.x];
    const InstInfo in = info[inst];
    if (!after_previous()) return;
    __shared__ DiagShared<R> sh;
    const int tid = threadIdx.x;
    if (status[inst] != ST_RUN) return;
    const int ld = dense_ld(in.m);
    const int k0 = s * kFb;
    const int nb = min(R, in.m - k0);
    double* A = dense + in.dn + (int64_t)k0 * ld + k0;
    const int col = tid % R, row = tid / R;
    double v[R / 4];
#pragma unroll
    for (int i = 0; i < R / 4; ++i) {
        const int rr = 4 * i + row;
        v[i] = (rr < nb && col <= rr) ? A[(int64_t)rr * ld + col] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < R / 4; ++i) sh.A[4 * i + row][col] = v[i];
    __syncthreads();
    const int r = tid % R, g = tid / R;
    double a[R / 16][4];
#pragma unroll
    for (int i = 0; i < R / 16; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[i][e] = sh.A[r][16 * i + 4 * g + e];
    if (tid < 16) sh.pb[tid >> 2][tid & 3] = sh.A[tid >> 2][tid & 3];
    __syncthreads();  // the columns of L overwrite sh.A
    double w[4];
    diag_rounds<0>(sh, a, w, nb, tol, r, g);
    if constexpr (R > 16) diag_rounds<1>(sh, a, w, nb, tol, r, g);
    if constexpr (R > 32) diag_rounds<2>(sh, a, w, nb, tol, r, g);
    if constexpr (R > 48) diag_rounds<3>(sh, a, w, nb, tol, r, g);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < R / 4; ++i) {
        const int rr = 4 * i + row;
        if (rr < nb && col < rr) A[(int64_t)rr * ld + col] = sh.A[rr][col];
    }
    if (tid < nb) dD[in.r0 + k0 + tid] = sh.d[tid];
}

// The entry of `cum` (inclusive cumulative counts of cnt instances) that item
// `idx` falls into.
__device__ __forceinline__ int item_instance(const int64_t* cum, int cnt, int64_t idx) {
    int lo = 0, hi = cnt - 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cum[mid] <= idx)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// L[r, k0:k1] = A[r, k0:k1] (L_blk D)^-T for kPanelT / G rows of one
// instance's panel per CTA: G neighbouring lanes share a row, each with every
// G-th pair of columns. A panel row exists only below a full block, so all 64
// columns are there. As soon as L[r, q] is final it is taken from every later
// column, which leaves independent updates in flight instead of one chain of
// subtractions per column; each element sees the same products in the same
// order (q ascending). The lanes of a row take column q from its owner by a
// shuffle and all form the quotient; a finished pair goes to shared memory, so
// a pair in which some lane still has a column left is updated in all of them.
// The columns go in two halves of 32 through the same code (a loop over the
// first half's columns, then the unrolled triangle): half the code of 64
// unrolled columns, which missed the instruction cache. The rows pass through
// shared memory (16-byte copies in, whole lines out) except the second half's
// way in, which there is no room for at three CTAs per SM.
// What bounds it is the latency of a row's 64 steps and the L1 data path (16
// bytes of L to every lane per four FP64 instructions). A lane per row has the
// fewest instructions and is the form for panels that fill the GPU: 954 us for
// the 17 such panels of 384 LPs of m 50-2000 (all 30: 1,163; 2,156 with a chain
// per column; 32 instead of 8 loads of L in flight give 4 of 100);
// with two rows for two lanes, which halves the loads of L, the iteration
// takes 8,081 us instead of 7,798, with four for four 9,007. Where a panel is
// small a warp's 4,000 FP64 instructions per row are its time, and four lanes
// per row take it from 16.6 to 13.2 us: an iteration of 48 LPs of m 50-300 takes
// 421 us instead of 450 (428 with eight lanes). The line: kPanelWide chunks,
// about one wave of the four-lane form's CTAs. The iteration of the 384 LPs,
// whose last panels are small, by the line: 7,798 us at none, 7,781 at 100,
// 7,798 at 160, 7,860 at 260, 8,295 at all.
constexpr int64_t kPanelWide = 100;
constexpr int kPanelT = 128;
constexpr int kPanelP = kFb + 2;  // even: 16-byte loads of two entries
constexpr int kHalf = kFb / 2;
constexpr int kRowP = kHalf + 2;  // staged rows: 16-byte accesses of eight lanes hit distinct banks
constexpr size_t panel_smem(int rows) { return sizeof(double) * (kFb * kPanelP + 2 * kFb + rows * kRowP); }

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

template <int G>
__global__ void __launch_bounds__(kPanelT, 3) batch_ldlt_panel_kernel(int s, const Chunk* __restrict__ chunks,
                                                                      const InstInfo* __restrict__ info,
                                                                      const int32_t* __restrict__ status, double* dense,
                                                                      const double* __restrict__ dD) {
    const Chunk ch = chunks[blockIdx.x / (kT / (kPanelT / G))];
    const InstInfo in = info[ch.inst];
    if (!after_previous()) return;
    constexpr int kRows = kPanelT / G, kPairs = kHalf / 2 / G;
    extern __shared__ __align__(16) double panel_sm[];
    double(*sLt)[kPanelP] = reinterpret_cast<double(*)[kPanelP]>(panel_sm);  // sLt[q][c] = L[k0 + c, k0 + q]
    double* sD = panel_sm + kFb * kPanelP;
    double* sY = sD + kFb;  // 1 / D, zero where a quotient needs the division
    double(*sRow)[kRowP] = reinterpret_cast<double(*)[kRowP]>(sY + kFb);  // half the columns of every row
    const int tid = threadIdx.x;
    if (status[ch.inst] != ST_RUN) return;
    const int ld = dense_ld(in.m);
    const int k0 = s * kFb;
    const int rb = k0 + kFb + ch.local * kT + static_cast<int>(blockIdx.x % (kT / kRows)) * kRows;
    const int rows = min(kRows, in.m - rb);
    if (rows <= 0) return;
    double* A = dense + in.dn;
    double* P = A + (int64_t)rb * ld + k0;  // the panel's rows
    const int piece = tid & 15, line = tid >> 4;  // copies: 16 lanes a row
#pragma unroll 4
    for (int r = line; r < rows; r += kPanelT / 16) cp_async16(&sRow[r][2 * piece], P + (int64_t)r * ld + 2 * piece);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
#pragma unroll
    for (int idx = tid; idx < kFb * kFb; idx += kPanelT) {
        const int rr = idx / kFb, c = idx % kFb;
        sLt[c][rr] = c < rr ? A[(int64_t)(k0 + rr) * ld + k0 + c] : 0.0;
    }
    if (tid < kFb) {
        const double d = dD[in.r0 + k0 + tid];
        sD[tid] = d;
        sY[tid] = divisor_reciprocal(d);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    // columns 2 (G i + side) and the next of a half belong to this lane
    const int side = tid % G;
    double* mine = sRow[tid / G];
    double v[2 * kPairs];
    auto load = [&](const double* from) {
#pragma unroll
        for (int i = 0; i < kPairs; ++i) {
            const double2 t = *reinterpret_cast<const double2*>(from + 2 * (G * i + side));
            v[2 * i] = t.x;
            v[2 * i + 1] = t.y;
        }
    };
    load(mine);
    __syncwarp();
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        if (h == 1) {
#pragma unroll 1
            for (int q = 0; q < kHalf; q += 2) {
                // L[r, q] D_q, rounded once as every column uses it
                const double2 lq = *reinterpret_cast<const double2*>(mine + q);
                const double w0 = lq.x * sD[q], w1 = lq.y * sD[q + 1];
                const double *l0 = &sLt[q][kHalf + 2 * side], *l1 = &sLt[q + 1][kHalf + 2 * side];
#pragma unroll
                for (int i = 0; i < kPairs; ++i) {
                    const double2 t = *reinterpret_cast<const double2*>(l0 + 2 * G * i);
                    const double2 u = *reinterpret_cast<const double2*>(l1 + 2 * G * i);
                    v[2 * i] -= w0 * t.x;
                    v[2 * i + 1] -= w0 * t.y;
                    v[2 * i] -= w1 * u.x;
                    v[2 * i + 1] -= w1 * u.y;
                }
            }
            __syncthreads();  // the first half has been used and has left sRow
        }
        const double* sLh = &sLt[h * kHalf][h * kHalf + 2 * side];
        double l[2];
#pragma unroll
        for (int q = 0; q < kHalf; ++q) {
            const int owner = q / 2 % G, i0 = q / 2 / G;
            const double d = sD[h * kHalf + q], y = sY[h * kHalf + q];
            double a = v[2 * i0 + q % 2];
            if (G > 1) a = __shfl_sync(0xffffffffu, a, owner, G);
            l[q % 2] = quotient(a, d, y);
            if (y == 0.0 || !(in_range(a) || a == 0.0)) l[q % 2] = a / d;
            const double w = l[q % 2] * d;
            if (q % 2 == 1 && side == owner) *reinterpret_cast<double2*>(mine + q - 1) = make_double2(l[0], l[1]);
            // finished columns of pair i0 take part and are not used again
#pragma unroll
            for (int i = i0; i < kPairs; ++i) {
                if (i == i0 && owner == G - 1 && q % 2 == 1) continue;
                const double2 t = *reinterpret_cast<const double2*>(sLh + q * kPanelP + 2 * G * i);
                v[2 * i] -= w * t.x;
                v[2 * i + 1] -= w * t.y;
            }
        }
        if (h == 0) load(P + (int64_t)min(tid / G, rows - 1) * ld + kHalf);
        // whole lines of half h of the rows
        __syncthreads();
#pragma unroll 4
        for (int r = line; r < rows; r += kPanelT / 16)
            *reinterpret_cast<double2*>(P + (int64_t)r * ld + h * kHalf + 2 * piece) =
                *reinterpret_cast<const double2*>(&sRow[r][2 * piece]);
    }
}

// Trailing update by NP (1 or 2) neighbouring 64-column panels at once:
// A[rows, cols] -= sum over the panels p of (L_p D_p) L_p^T, in 64 x 64 tiles
// spread over persistent CTAs, two per SM (one multiplies while the other
// changes tiles). Two panels per visit halve the reads and writes of the
// trailing matrix, which is far larger than L2. A producer warp finds the
// tiles (a chain of dependent loads) and copies the panels in slices of 16
// columns into a ring of kUpdStages stages that runs on across tiles, and the
// output tile with a slice of the first panel; 4 consumer warps multiply.
// Everything is handed over with named barriers: no polling. How far the
// producer is ahead decides the rate, so rows are packed and swizzled by
// 16-byte pieces instead of padded, to fit a fifth stage; output tiles read
// straight into registers at the tile's start held the products up. A consumer
// warp owns 32 x 32 of the tile: per 4 columns 8 fragment loads feed 16 DMMAs.
// D is applied at the fragment load (a = L[r, k] D_k rounds once). An
// element's accumulator starts at zero for every panel and is subtracted after
// it, so it goes through the same operations in the same order whatever the
// grouping of the panels. Rows past m keep what the stage held before: they
// only reach outputs past m.
// 384 LPs of m 50-2000: 3,797 us (2,650 at the FP64 tensor rate of 37 TFLOP/s);
// 5,641 with one panel per visit and one commit group ahead. Products alone
// take 2,780 us of that, the copies alone 2,720.
constexpr int kUpdN = kFb, kUpdK = 16;         // tile edge, columns of a slice
constexpr int kUpdWarps = 4;                   // consumers
constexpr int kUpdT = 32 * (kUpdWarps + 1);    // and the producer warp
constexpr int kUpdStages = 5;
constexpr int kUpdAhead = 3;                   // slices in flight when one is handed over
constexpr int kUpdStage = 2 * kUpdN * kUpdK + kUpdK;  // doubles: A rows, B rows, D
constexpr size_t kUpdSmem = sizeof(double) * (kUpdStages * kUpdStage + kUpdN * kUpdN);
static_assert(2 * (kUpdSmem + 1280) <= 228 * 1024, "two update CTAs per SM");

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}

// Whole warps meet here (bar.sync and bar.arrive are .aligned), after branches by lane as well.
__device__ __forceinline__ void named_sync(int id) {
    __syncwarp();
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "n"(kUpdT) : "memory");
}
__device__ __forceinline__ void named_arrive(int id) {
    __syncwarp();
    asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "n"(kUpdT) : "memory");
}

// 64 x 64 tiles of a trailing matrix of T block rows: its lower triangle, or its first block column.
__host__ __device__ __forceinline__ int64_t update_tiles(int64_t T, bool column) {
    return column ? T : T * (T + 1) / 2;
}

struct UpdTile {
    double* A;  // the instance's dense block, null: no more tiles
    int m, ld, rb, cb;
};

template <int NP>
__global__ void __launch_bounds__(kUpdT, 2) batch_ldlt_update_kernel(int k0, int kt, int column, int cnt, int64_t ntiles,
                                                                  const int64_t* __restrict__ tiles,
                                                                  const InstInfo* __restrict__ info,
                                                                  const int32_t* __restrict__ order,
                                                                  const int32_t* __restrict__ status,
                                                                  double* __restrict__ dense,
                                                                  const double* __restrict__ dD) {
    extern __shared__ __align__(16) double upd_smem[];
    __shared__ UpdTile s_tile[kUpdStages];
    double* sC = upd_smem + kUpdStages * kUpdStage;
    constexpr int kPanel = kFb / kUpdK;  // slices of a panel
    constexpr int kSlices = NP * kPanel;  // slices of a tile
    constexpr int kFull = 1, kEmpty = 1 + kUpdStages, kOut = 1 + 2 * kUpdStages;  // named barriers: stages, output tile
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (warp == kUpdWarps) {
        bool out_used = false;  // the consumers still have to release the output tile
        int64_t n = 0;  // slices issued; slice i goes to stage i mod kUpdStages
        int b = item_instance(tiles, cnt, blockIdx.x);
        int inst = order[min(b, cnt - 1)];
        InstInfo in = info[inst];
        if (!after_previous()) return;
        for (int64_t idx = blockIdx.x; idx < ntiles; idx += gridDim.x) {
            if (idx != blockIdx.x) {
                b = item_instance(tiles, cnt, idx);
                inst = order[b];
                in = info[inst];
            }
            if (status[inst] != ST_RUN) continue;
            const int64_t local = idx - (b > 0 ? tiles[b - 1] : 0);
            int I = static_cast<int>(local), J = 0;
            if (!column) {
                I = static_cast<int>((sqrt(8.0 * (double)local + 1.0) - 1.0) * 0.5);
                while ((int64_t)(I + 1) * (I + 2) / 2 <= local) ++I;
                while ((int64_t)I * (I + 1) / 2 > local) --I;
                J = static_cast<int>(local - (int64_t)I * (I + 1) / 2);
            }
            UpdTile t;
            t.m = in.m;
            t.ld = dense_ld(t.m);
            t.rb = kt + I * kUpdN;
            t.cb = kt + J * kUpdN;
            t.A = dense + in.dn;
            // a lane copies 16-byte piece `lane mod 8` of every fourth row;
            // piece c of row r lies at c ^ (r mod 8)
            const int quad = lane >> 3, piece = lane & 7;
            const int nA = min(kUpdN, t.m - t.rb), nB = min(kUpdN, t.m - t.cb);
            const int64_t step = 4 * (int64_t)t.ld;
            auto copy_rows = [&](double* dst, int row0, int n, int kc) {
                const double* src = t.A + (int64_t)(row0 + quad) * t.ld + kc + 2 * piece;
#pragma unroll 8
                for (int r = quad; r < n; r += 4, src += step)
                    cp_async16(dst + r * kUpdK + 2 * (piece ^ (r & 7)), src);
            };
            for (int h = 0; h < kSlices; ++h, ++n) {
                const int st = static_cast<int>(n % kUpdStages);
                if (n >= kUpdStages) named_sync(kEmpty + st);
                double* base = upd_smem + st * kUpdStage;
                const int kc = k0 + h * kUpdK;
                copy_rows(base, t.rb, nA, kc);
                copy_rows(base + kUpdN * kUpdK, t.cb, nB, kc);
                if (lane < kUpdK) cp_async8(base + 2 * kUpdN * kUpdK + lane, dD + in.r0 + kc + lane);
                if (h == kPanel - 1) {
                    if (out_used) named_sync(kOut);
                    out_used = true;
                    // piece c of output row r lies at c ^ 4 (r mod 2)
                    if (t.cb + 2 * lane < t.m) {
                        const double* src = t.A + (int64_t)t.rb * t.ld + t.cb + 2 * lane;
#pragma unroll 8
                        for (int r = 0; r < nA; ++r, src += t.ld)
                            cp_async16(sC + r * kUpdN + 2 * (lane ^ ((r & 1) << 2)), src);
                    }
                }
                if (lane == 0) s_tile[st] = t;
                asm volatile("cp.async.commit_group;\n" ::: "memory");
                if (n >= kUpdAhead) {  // slice n - kUpdAhead has arrived
                    asm volatile("cp.async.wait_group %0;\n" ::"n"(kUpdAhead) : "memory");
                    named_arrive(kFull + static_cast<int>((n - kUpdAhead) % kUpdStages));
                }
            }
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        for (int64_t i = n >= kUpdAhead ? n - kUpdAhead : 0; i < n; ++i) named_arrive(kFull + static_cast<int>(i % kUpdStages));
        // the end mark, then every barrier the consumers still arrive at
        const int st = static_cast<int>(n % kUpdStages);
        if (n >= kUpdStages) named_sync(kEmpty + st);
        if (lane == 0) s_tile[st].A = nullptr;
        named_arrive(kFull + st);
        for (int64_t i = n >= kUpdStages ? n - kUpdStages + 1 : 0; i < n; ++i)
            named_sync(kEmpty + static_cast<int>(i % kUpdStages));
        if (out_used) named_sync(kOut);
        return;
    }
    if (!after_previous()) return;
    const int wr = (warp >> 1) * 32, wc = (warp & 1) * 32;
    const int fr = lane >> 2, fk = lane & 3, sw = (fk >> 1) ^ fr;
    int st = 0;
    for (;;) {
        named_sync(kFull + st);
        const UpdTile t = s_tile[st];
        if (!t.A) return;
        // this lane's output elements: rows gr(i), column pairs gc(j), gc(j) + 1
        double c[4][4][2];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            double acc[4][4][2];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll 1
            for (int h = 0; h < kPanel; ++h) {
                if (p + h > 0) named_sync(kFull + st);
                const double* sA = upd_smem + st * kUpdStage + (wr + fr) * kUpdK;
                const double* sB = upd_smem + st * kUpdStage + (kUpdN + wc + fr) * kUpdK;
                const double* sD = upd_smem + st * kUpdStage + 2 * kUpdN * kUpdK + fk;
#pragma unroll
                for (int kq = 0; kq < kUpdK; kq += 4) {
                    const int at = 2 * ((kq >> 1) ^ sw) + (fk & 1);  // column kq + fk of a row = fr mod 8
                    const double dk = sD[kq];
                    double a[4], b[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) a[i] = sA[8 * i * kUpdK + at] * dk;  // A(8x4)[fr][fk]
#pragma unroll
                    for (int j = 0; j < 4; ++j) b[j] = sB[8 * j * kUpdK + at];  // B(4x8)[fk][fr]
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j) dmma_m8n8k4(acc[i][j], a[i], b[j]);
                }
                named_arrive(kEmpty + st);
                st = (st + 1) % kUpdStages;
            }
            const double* o = sC + (wr + fr) * kUpdN + wc + 2 * fk;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (p == 0) {
                        const double2 v = *reinterpret_cast<const double2*>(o + 8 * i * kUpdN + 8 * (j ^ (fr & 1)));
                        c[i][j][0] = v.x;
                        c[i][j][1] = v.y;
                    }
                    c[i][j][0] -= acc[i][j][0];
                    c[i][j][1] -= acc[i][j][1];
                }
            if (p == 0) named_arrive(kOut);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int gr = t.rb + wr + 8 * i + fr;
            if (gr >= t.m) continue;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int gc = t.cb + wc + 8 * j + 2 * fk;
                double* o = t.A + (int64_t)gr * t.ld + gc;
                if (gc < gr)
                    *reinterpret_cast<double2*>(o) = make_double2(c[i][j][0], c[i][j][1]);
                else if (gc == gr)
                    *o = c[i][j][0];
            }
        }
    }
}

// ---- batched triangular solves: N_i x = b in place, N_i = L_i D_i L_i^T ----
// One launch per solve. An instance belongs to one CTA, which then keeps its
// vector in shared memory, or to 2, 4 or 8 CTAs of a cluster; the CTAs walk
// its 64-row blocks together, forward and then backward, one cluster barrier
// per block. (A launch per block and direction spent 8 us and more each on
// starting, finding its place and draining, for microseconds of products.)
//   forward : every CTA solves the unit-lower diagonal block itself (64 steps
//     of one warp) and takes the block's contribution from its chunks' right-
//     hand sides, in place; the first CTA keeps the block of y / D in `work`.
//   backward: every CTA forms its chunks' column-block dot products of L^T x;
//     after the barrier the first CTA sums them in chunk order and solves the
//     diagonal block while the others go on to the next block's products.
//     (Only the first chunk of the next block touches the solution it writes,
//     and that chunk is the first CTA's; the others reach it blocks later.)
// Rows below a block come in chunks of kT, chunk c to CTA c mod the group's
// size. L does not depend on x, so each warp's next 16 rows and the next
// diagonal block load ahead of the barriers. Every sum has a fixed order
// whatever the group size: a row's forward sum is a butterfly over the lanes;
// a backward sum runs over a warp's rows (every eighth of the chunk), then
// the warps, then the chunks.
// An instance takes part when it is iterating and, with a refine mask, still
// refining.
// A warp takes 16 rows of a chunk, then 16 of its second half, so that chunks
// of up to 128 rows are one batch, and the quotients by D are formed beside the
// products: 36 us a solve of 48 LPs of m 50-300, 42 with 32 rows in a run and
// the quotients before them. 384 LPs of m 50-2000, both solves of an
// iteration: 1,075 us; 3,853 with a launch per block (the factors alone are 3
// GB of reads, 470 us).
__device__ __forceinline__ bool solving(const int32_t* status, const int32_t* refine, int inst) {
    return status[inst] == ST_RUN && (!refine || refine[inst]);
}

constexpr int kSolveCluster = 8;
constexpr int kSolveRows = 16;                      // rows of L a warp has in flight
constexpr int kSolveBatches = kT / 8 / kSolveRows;  // such batches of a warp per chunk
constexpr int kSolveP = kFb + 2;                    // smem row stride: 16-byte copies

// One butterfly level over lane bit o of 2 R partial sums per lane: a lane
// keeps the R sums of its half and adds its partner's, own + partner as the
// one-sum butterfly adds them.
template <int R>
__device__ __forceinline__ void fold(double* p, int lane, int o) {
    const bool up = lane & o;
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const double keep = up ? p[u + R] : p[u], give = up ? p[u] : p[u + R];
        p[u] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
}

__device__ __forceinline__ double ld_l2(const double* p) {  // written by other CTAs: past L1
    double v;
    asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ double ld_once(const double* p) {  // in program order, so that the batch stays in flight
    double v;
    asm volatile("ld.global.cs.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// The strictly lower part of the diagonal block at k0 (rows below m only), asynchronously.
__device__ __forceinline__ void copy_diag_block(double (*sL)[kSolveP], const double* L, int ld, int k0, int nb) {
#pragma unroll
    for (int q = 0; q < kFb * kFb / 2 / kT; ++q) {
        const int u = threadIdx.x + q * kT, r = u / (kFb / 2), c = 2 * (u % (kFb / 2));
        if (r < nb && c < r) cp_async16(&sL[r][c], L + (int64_t)(k0 + r) * ld + k0 + c);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// y = L^-1 v of a unit-lower diagonal block by one warp, rows lane and lane + 32
// (v0, v1), four columns per step: every lane solves the 4 x 4 corner itself
// from four broadcasts. Unrolled in full, so that the loads of L run ahead of
// the chain (3,130 cycles; 4,700 in a loop, 3,450 with a broadcast per column,
// unrolled by 8). A row takes its columns in order. Rows past the block only
// reach themselves and later ones.
__device__ __forceinline__ void forward_block(const double (*sL)[kSolveP], double& v0, double& v1, int lane) {
#pragma unroll
    for (int j = 0; j < kFb; j += 4) {
        double y[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) y[q] = __shfl_sync(0xffffffffu, j < 32 ? v0 : v1, (j + q) & 31);
#pragma unroll
        for (int q = 0; q < 3; ++q)
#pragma unroll
            for (int e = q + 1; e < 4; ++e) y[e] -= sL[j + e][j + q] * y[q];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (j < 32 && lane > j + q) v0 -= sL[lane][j + q] * y[q];
            if (j < 32 || lane + 32 > j + q) v1 -= sL[lane + 32][j + q] * y[q];
        }
    }
}

// x = L^-T v likewise, columns descending. Rows past the instance's last one
// are zero in L and v and change nothing.
__device__ __forceinline__ void backward_block(const double (*sL)[kSolveP], double& v0, double& v1, int lane) {
#pragma unroll
    for (int j = kFb - 1; j >= 0; j -= 4) {
        double y[4];  // entries j, j - 1, j - 2, j - 3
#pragma unroll
        for (int q = 0; q < 4; ++q) y[q] = __shfl_sync(0xffffffffu, j < 32 ? v0 : v1, (j - q) & 31);
#pragma unroll
        for (int q = 0; q < 3; ++q)
#pragma unroll
            for (int e = q + 1; e < 4; ++e) y[e] -= sL[j - q][j - e] * y[q];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (j >= 32 || lane < j - q) v0 -= sL[j - q][lane] * y[q];
            if (j >= 32 && lane + 32 < j - q) v1 -= sL[j - q][lane + 32] * y[q];
        }
    }
}

// The same for batches whose instances have one block each: a warp per
// instance, R the largest one's rows (16, 32 or 64). Few are bound by the
// launch and the chain, many by how many an SM holds: a CTA of the kernel below
// takes a quarter of the SM and a full block's steps for them. hn_batch_solve of
// 16,000 instances of 10 rows takes 97 us, of 32 rows 181, of 64 rows 420 (506,
// 605 and 687 below; 248, 458 and 733 with a launch per direction); of one
// instance of 10 rows 22, of 64 rows 28 (28 and 28.5 below).
template <int R>
__global__ void __launch_bounds__(32) batch_solve_block_kernel(const InstInfo* __restrict__ info,
                                                               const int32_t* __restrict__ status,
                                                               const int32_t* __restrict__ refine,
                                                               const double* __restrict__ dense,
                                                               const double* __restrict__ dD, double* xv) {
    const InstInfo in = info[blockIdx.x];
    if (!after_previous()) return;
    if (!solving(status, refine, blockIdx.x)) return;
    __shared__ double sL[R][R + 1];
    const int lane = threadIdx.x, m = in.m, ld = dense_ld(m);
    const double* L = dense + in.dn;
    double* x = xv + in.r0;
    constexpr int kBatch = R < 32 ? R * R / 32 : 16;  // loads in flight
#pragma unroll 1
    for (int q0 = 0; q0 < R * R / 32 && q0 * 32 < m * R; q0 += kBatch) {
        double t[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
            const int r = (32 * (q0 + q) + lane) / R, c = lane % R + (R > 32 ? 32 * ((q0 + q) % (R / 32)) : 0);
            t[q] = r < m && c < r ? L[(int64_t)r * ld + c] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
            const int r = (32 * (q0 + q) + lane) / R, c = lane % R + (R > 32 ? 32 * ((q0 + q) % (R / 32)) : 0);
            sL[r][c] = t[q];
        }
    }
    const bool on0 = lane < m, on1 = R > 32 && lane + 32 < m;
    double v0 = on0 ? x[lane] : 0.0, v1 = on1 ? x[lane + 32] : 0.0;
    const double d0 = on0 ? dD[in.r0 + lane] : 1.0, d1 = on1 ? dD[in.r0 + lane + 32] : 1.0;
    __syncwarp();
#pragma unroll 4
    for (int j = 0; j < m; ++j) {
        const double y = __shfl_sync(0xffffffffu, R > 32 && j >= 32 ? v1 : v0, j & 31);
        if (on0 && lane > j) v0 -= sL[lane][j] * y;
        if (on1 && lane + 32 > j) v1 -= sL[lane + 32][j] * y;
    }
    v0 /= d0;
    v1 /= d1;
#pragma unroll 4
    for (int j = m - 1; j >= 0; --j) {
        const double y = __shfl_sync(0xffffffffu, R > 32 && j >= 32 ? v1 : v0, j & 31);
        if (lane < j) v0 -= sL[j][lane] * y;
        if (R > 32 && lane + 32 < j) v1 -= sL[j][lane + 32] * y;
    }
    if (on0) x[lane] = v0;
    if (on1) x[lane + 32] = v1;
}

__global__ void __cluster_dims__(kSolveCluster, 1, 1) __launch_bounds__(kT, 2)
    batch_solve_kernel(const SolveSlot* __restrict__ slots, const InstInfo* __restrict__ info,
                       const int32_t* __restrict__ status, const int32_t* __restrict__ refine,
                       const double* __restrict__ dense, const double* __restrict__ dD, double* work, double* part,
                       double* xv) {
    const SolveSlot slot = slots[blockIdx.x];
    InstInfo in = {0, 0, 0, {0, 0, 0}};
    if (slot.inst >= 0) in = info[slot.inst];
    if (!after_previous()) return;
    extern __shared__ __align__(16) double solve_smem[];
    double(*sLb)[kFb][kSolveP] = reinterpret_cast<double(*)[kFb][kSolveP]>(solve_smem);  // two diagonal blocks
    double* s_x = solve_smem + 2 * kFb * kSolveP;  // a single CTA's instance: right-hand side, y / D, solution
    __shared__ double sacc[kT / 32][kFb];
    __shared__ double sx[kFb];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (slot.inst >= 0 && !solving(status, refine, slot.inst)) in = {0, 0, 0, {0, 0, 0}};
    const int m = in.m, ld = dense_ld(m);
    const double* L = dense + in.dn;
    double* x = xv + in.r0;
    double* y = work + in.r0;
    const double* D = dD + in.r0;
    const int nblk = (m + kFb - 1) / kFb;
    const bool alone = slot.size == 1;
    const int steps = slot.steps > 0 ? slot.steps : nblk;
    if (alone)
        for (int i = tid; i < m; i += kT) s_x[i] = x[i];
    auto barrier = [&]() {
        if (slot.steps > 0) {
            __syncwarp();  // .aligned, and rows past the instance's end branch by lane
            asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
        } else {
            __syncthreads();
        }
    };
    double p0[kSolveRows], p1[kSolveRows];

    // ---- forward ----
    // batch h of this warp's rows in chunk c below the block at k0: rows first, first + 1, ...
    auto fwd_row = [&](int k0, int c, int h) {
        return k0 + kFb + c * kT + h * kSolveRows * (kT / 32) + warp * kSolveRows;
    };
    auto fwd_load = [&](int k0, int c, int h) {
        const int r = fwd_row(k0, c, h);
#pragma unroll
        for (int u = 0; u < kSolveRows; ++u) {
            p0[u] = p1[u] = 0.0;
            if (r + u < m) {
                const double* Lr = L + (int64_t)(r + u) * ld + k0;
                p0[u] = ld_once(Lr + lane);
                p1[u] = ld_once(Lr + lane + 32);
            }
        }
    };
    if (nblk > 0) {
        copy_diag_block(sLb[0], L, ld, 0, min(kFb, m));
        fwd_load(0, slot.rank, 0);
    }
    for (int s = 0; s < steps; ++s) {
        if (s < nblk) {
            const int k0 = s * kFb, nb = min(kFb, m - k0);
            const auto sL = sLb[s & 1];
            // the other buffer was last read a barrier ago
            if (s + 1 < nblk)
                copy_diag_block(sLb[(s + 1) & 1], L, ld, k0 + kFb, min(kFb, m - k0 - kFb));
            else
                asm volatile("cp.async.commit_group;\n" ::: "memory");
            // a lane's share of each row batch: row first + mine
            const int mine = (lane >> 1);
            double xr = 0.0;
            // y / D is formed beside the products, by the warps that more often have no rows
            const int dr = tid - (kT - kFb);
            const bool divides = slot.rank == 0 && dr >= 0 && dr < nb;
            const double d = divides ? D[k0 + dr] : 0.0;
            if (!alone) {
                const int r = fwd_row(k0, slot.rank, 0) + mine;
                if (r < m) xr = ld_l2(x + r);
                if (tid < kFb) sx[tid] = tid < nb ? ld_l2(x + k0 + tid) : 0.0;
            }
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncthreads();
            if (warp == 0) {
                double v0, v1;
                if (alone) {
                    v0 = lane < nb ? s_x[k0 + lane] : 0.0;
                    v1 = lane + 32 < nb ? s_x[k0 + lane + 32] : 0.0;
                } else {
                    v0 = sx[lane];
                    v1 = sx[lane + 32];
                }
                forward_block(sL, v0, v1, lane);
                sx[lane] = v0;
                sx[lane + 32] = v1;
            }
            __syncthreads();
            if (divides) (alone ? s_x : y)[k0 + dr] = sx[dr] / d;
            const double x0 = sx[lane], x1 = sx[lane + 32];
            for (int c = slot.rank; k0 + kFb + c * kT < m; c += slot.size) {
#pragma unroll 1
                for (int h = 0;; ++h) {
                    double p[kSolveRows];
#pragma unroll
                    for (int u = 0; u < kSolveRows; ++u) p[u] = p0[u] * x0 + p1[u] * x1;
                    const int row = fwd_row(k0, c, h) + mine;
                    const double old = alone ? (row < m ? s_x[row] : 0.0) : xr;
                    const bool more = h + 1 < kSolveBatches && fwd_row(k0, c, h + 1) < m;
                    const int nc = more ? c : c + slot.size, nh = more ? h + 1 : 0;
                    if (k0 + kFb + nc * kT < m) {
                        fwd_load(k0, nc, nh);
                        const int r = fwd_row(k0, nc, nh) + mine;
                        if (!alone && r < m) xr = ld_l2(x + r);
                    } else {
                        fwd_load(k0 + kFb, slot.rank, 0);
                    }
                    fold<8>(p, lane, 16);
                    fold<4>(p, lane, 8);
                    fold<2>(p, lane, 4);
                    fold<1>(p, lane, 2);
                    double t = p[0];
                    t = t + __shfl_xor_sync(0xffffffffu, t, 1);
                    if (!(lane & 1) && row < m) (alone ? s_x : x)[row] = old - t;
                    if (!more) break;
                }
            }
        }
        barrier();
    }

    // ---- backward ----
    // batch h of this warp's rows in chunk c below the block at k0: rows first, first + 8, ...
    auto bwd_row = [&](int k0, int c, int h) { return k0 + kFb + c * kT + warp + h * kSolveRows * (kT / 32); };
    auto bwd_load = [&](int k0, int c, int h) {
        const int r = bwd_row(k0, c, h);
#pragma unroll
        for (int u = 0; u < kSolveRows; ++u) {
            p0[u] = p1[u] = 0.0;
            if (r + u * (kT / 32) < m) {
                const double* Lr = L + (int64_t)(r + u * (kT / 32)) * ld + k0;
                p0[u] = ld_once(Lr + lane);
                p1[u] = ld_once(Lr + lane + 32);
            }
        }
    };
    // this instance's partial sums: chunk c of an even (odd) block at part_i + 64 c (+ half)
    const int64_t half = 64 * (int64_t)((m + kT - 1) / kT);
    double* part_i = part + 2 * 64 * (in.r0 / kT + (slot.inst >= 0 ? slot.inst : 0));
    int s = nblk - 1;
    if (s >= 0) {
        if (slot.rank == 0) {
            for (int u = (m - s * kFb) * kFb + tid; u < kFb * kFb; u += kT) sLb[s & 1][u / kFb][u % kFb] = 0.0;
            copy_diag_block(sLb[s & 1], L, ld, s * kFb, m - s * kFb);
        }
        bwd_load(s * kFb, slot.rank, 0);
    }
    for (int i = 0; i < steps; ++i, --s) {
        double* ps = part_i + (s & 1) * half;
        const int k0 = s * kFb;
        const auto sL = sLb[s & 1];
        if (slot.rank == 0) {  // as forward; only the first CTA solves
            if (s > 0)
                copy_diag_block(sLb[(s - 1) & 1], L, ld, k0 - kFb, kFb);
            else
                asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
        const int nch = s >= 0 ? (max(0, m - k0 - kFb) + kT - 1) / kT : 0;
        double t = 0.0;
        for (int c = slot.rank; c < nch; c += slot.size) {
            double a0 = 0.0, a1 = 0.0;
#pragma unroll 1
            for (int h = 0;; ++h) {
                const int r = bwd_row(k0, c, h);
                double xc[kSolveRows];
#pragma unroll
                for (int u = 0; u < kSolveRows; ++u) {
                    const int row = r + u * (kT / 32);
                    xc[u] = 0.0;
                    if (row < m) xc[u] = alone ? s_x[row] : ld_l2(x + row);
                }
#pragma unroll
                for (int u = 0; u < kSolveRows; ++u) {
                    const bool row = r + u * (kT / 32) < m;
                    const double t0 = a0 + p0[u] * xc[u], t1 = a1 + p1[u] * xc[u];
                    a0 = row ? t0 : a0;
                    a1 = row ? t1 : a1;
                }
                const bool more = h + 1 < kSolveBatches && bwd_row(k0, c, h + 1) < m;
                if (more)
                    bwd_load(k0, c, h + 1);
                else if (c + slot.size < nch)
                    bwd_load(k0, c + slot.size, 0);
                else if (s > 0)
                    bwd_load(k0 - kFb, slot.rank, 0);
                if (!more) break;
            }
            sacc[warp][lane] = a0;
            sacc[warp][lane + 32] = a1;
            __syncthreads();
            if (tid < kFb) {
                t = 0.0;
                for (int w = 0; w < kT / 32; ++w) t += sacc[w][tid];
                if (nch > 1) ps[64 * c + tid] = t;  // read back by this thread, or past the barrier
            }
            __syncthreads();
        }
        if (slot.rank >= nch && s > 0) bwd_load(k0 - kFb, slot.rank, 0);  // no chunk here, maybe at the next block
        barrier();
        if (s >= 0 && slot.rank == 0) {
            const int nb = min(kFb, m - k0);
            if (tid < kFb) {
                if (nch > 1) {
                    t = 0.0;
                    for (int c = 0; c < nch; ++c) t += ld_l2(ps + 64 * c + tid);
                }
                sx[tid] = tid < nb ? (alone ? s_x[k0 + tid] : y[k0 + tid]) - t : 0.0;
            }
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncthreads();
            if (warp == 0) {
                double v0 = sx[lane], v1 = sx[lane + 32];
                backward_block(sL, v0, v1, lane);
                double* o = alone ? s_x : x;
                if (lane < nb) o[k0 + lane] = v0;
                if (lane + 32 < nb) o[k0 + lane + 32] = v1;
            }
            __syncthreads();
        }
    }
    if (alone)
        for (int i = tid; i < m; i += kT) x[i] = s_x[i];  // past the last block's barrier
}

// Refinement bookkeeping per instance (refinement.cpp:15-30): with r = rhs - N x,
// rel = max|r| / max|rhs|; an instance keeps sweeping while rel > 1e-10 and
// sweeps remain; a sweeping instance's r is then solved and added to x. The
// start copies the right-hand sides into x; the check's last block puts the
// number of sweeping instances where the host reads it and clears the counts
// (nref[0] and nref[1], the blocks that have counted). Copies and fills of
// their own for these, with one in the assembly, took 34 us of the 421 of an
// iteration of 48 LPs of m 50-300.
__global__ void __launch_bounds__(kT) batch_refine_check_kernel(const int64_t* __restrict__ row_off,
                                                                const int32_t* __restrict__ status,
                                                                const double* __restrict__ rhs,
                                                                const double* __restrict__ ax, double* __restrict__ r,
                                                                int32_t* __restrict__ refine, int32_t* nref,
                                                                int32_t* left_host) {
    if (!after_previous()) return;
    __shared__ double sh[32];
    const int64_t i = blockIdx.x;
    if (status[i] == ST_RUN && refine[i]) {
        const int64_t r0 = row_off[i], r1 = row_off[i + 1];
        double nb = 0.0, nr = 0.0;
        for (int64_t k = r0 + threadIdx.x; k < r1; k += kT) {
            const double b = rhs[k], d = b - ax[k];
            nb = fmax(nb, fabs(b));
            nr = fmax(nr, fabs(d));
            r[k] = d;
        }
        nb = block_max<kT>(nb, sh);
        nr = block_max<kT>(nr, sh);
        if (threadIdx.x == 0) {
            const bool go = nb != 0.0 && nb == nb && nr / nb > 1e-10;
            refine[i] = go ? 1 : 0;
            if (go) atomicAdd(nref, 1);
        }
    }
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(nref + 1, 1) == static_cast<int32_t>(gridDim.x) - 1) {
            *left_host = atomicExch(nref, 0);
            nref[1] = 0;
        }
    }
}

__global__ void __launch_bounds__(kT) batch_refine_start_kernel(const int64_t* __restrict__ row_off,
                                                                const int32_t* __restrict__ status,
                                                                const double* rhs, int32_t* __restrict__ refine,
                                                                double* x) {
    if (!after_previous()) return;
    __shared__ double sh[32];
    const int64_t i = blockIdx.x;
    const int64_t r0 = row_off[i], r1 = row_off[i + 1];
    double nb = 0.0;
    for (int64_t k = r0 + threadIdx.x; k < r1; k += kT) {
        const double v = rhs[k];
        x[k] = v;
        nb = fmax(nb, fabs(v));
    }
    nb = block_max<kT>(nb, sh);
    // a zero or NaN right-hand side is not refined (refinement.cpp:17-18); fmax drops NaN,
    // so look for one explicitly
    __shared__ int s_nan;
    if (threadIdx.x == 0) s_nan = 0;
    __syncthreads();
    for (int64_t k = r0 + threadIdx.x; k < r1; k += kT)
        if (rhs[k] != rhs[k]) s_nan = 1;
    __syncthreads();
    if (threadIdx.x == 0) refine[i] = (status[i] == ST_RUN && nb != 0.0 && !s_nan) ? 1 : 0;
}

__global__ void batch_axpy_masked_kernel(int64_t m, const int32_t* __restrict__ row_inst,
                                         const int32_t* __restrict__ status, const int32_t* __restrict__ refine,
                                         const double* __restrict__ r, double* __restrict__ x) {
    if (!after_previous()) return;
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= m) return;
    const int inst = row_inst[k];
    if (status[inst] == ST_RUN && refine[inst]) x[k] += r[k];
}

__global__ void row_inst_kernel(int64_t K, const int64_t* __restrict__ row_off, int32_t* __restrict__ row_inst) {
    if (!after_previous()) return;
    const int64_t i = blockIdx.x;
    for (int64_t r = row_off[i] + threadIdx.x; r < row_off[i + 1]; r += blockDim.x) row_inst[r] = (int32_t)i;
}

__global__ void narrow_rp_kernel(int64_t n, const int64_t* __restrict__ in, int32_t* __restrict__ out) {
    if (!after_previous()) return;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = static_cast<int32_t>(in[i]);
}

void free_batch(hn_batch* B) {
    if (!B) return;
    dfree({B->row_off, B->col_off, B->row_inst, B->dn_off, B->order, B->dense, B->dD, B->refine, B->nref, B->nrp,
           B->tile_row, B->tile_nz, B->carry_row, B->head_row, B->carry_val, B->head_val, B->r, B->ax, B->step_tiles,
           B->chunks, B->info, B->slots, B->work, B->solve_part, B->kkt, B->kkt_ref, B->ref_iter, B->xb, B->zb,
           B->lb});
    host_word_free(B->left_host);
    delete B;
}

KktArgs kkt_args(const hn_batch* B, const double* lam, const double* b, const double* c) {
    return KktArgs{lam,    b,      c,      B->ru,  B->cu,       B->offset, B->kkt,
                   B->kkt_ref, B->xb, B->zb, B->lb, B->ref_iter, B->kkt_tol, B->kkt_extra};
}

SpmvMat n_mat(const hn_batch* B, const double* nval) {
    SpmvMat N{(int)B->m, (int)B->P->nnz, B->nrp, B->P->ci, nval, B->tile_row, B->tile_nz, B->carry_row,
              B->carry_val, B->head_row, B->head_val, B->ntiles};
    N.ticket = reinterpret_cast<unsigned*>(B->carry_row + B->ntiles);
    N.short_heads = B->short_heads;
    return N;
}

// x holds the right-hand sides of the taking-part instances on entry, their solutions on return.
void solve_all(hn_batch* B, const int32_t* status, const int32_t* refine, double* x, cudaStream_t s) {
    if (B->mmax <= kFb) {
        auto* kernel = B->mmax <= 16   ? batch_solve_block_kernel<16>
                       : B->mmax <= 32 ? batch_solve_block_kernel<32>
                                       : batch_solve_block_kernel<64>;
        launch_next(kernel, (unsigned)B->K, 32, 0, s, B->info, status, refine, B->dense, B->dD, x);
        launched("batch_solve_block_kernel");
        return;
    }
    launch_next(batch_solve_kernel, (unsigned)B->nslots, kT, (size_t)B->solve_smem, s, B->slots, B->info, status,
                refine, B->dense, B->dD, B->work, B->solve_part, x);
    launched("batch_solve_kernel");
}

}  // namespace
}  // namespace hn

using namespace hn;

extern "C" {

int hn_batch_create(int64_t K, const int64_t* row_off_host, const int64_t* col_off_host, const hn_pattern* P,
                    hn_batch** out) {
    return guard("hn_batch_create", [&] {
        require_init();
        if (K <= 0 || !row_off_host || !col_off_host || !P || !out) fail(HN_ERR_INVALID_ARG, "bad arguments");
        *out = nullptr;
        const int64_t m = row_off_host[K], n = col_off_host[K];
        if (m != P->m) fail(HN_ERR_INVALID_ARG, "row offsets do not match the pattern");
        std::vector<int64_t> dn(K + 1, 0);
        std::vector<int32_t> order(K);
        for (int64_t i = 0; i < K; ++i) {
            const int64_t mi = row_off_host[i + 1] - row_off_host[i];
            const int64_t ni = col_off_host[i + 1] - col_off_host[i];
            if (mi < 1 || ni < 1) fail(HN_ERR_INVALID_ARG, "every instance needs a row and a column");
            dn[i + 1] = dn[i] + mi * dense_ld(static_cast<int>(mi));
            order[i] = static_cast<int32_t>(i);
        }
        std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) {
            return row_off_host[a + 1] - row_off_host[a] > row_off_host[b + 1] - row_off_host[b];
        });
        hn_batch* B = new hn_batch();
        cudaStream_t s = nullptr;
        try {
            B->K = K;
            B->m = m;
            B->n = n;
            B->P = P;
            B->row_off = dmalloc<int64_t>(K + 1);
            B->col_off = dmalloc<int64_t>(K + 1);
            B->dn_off = dmalloc<int64_t>(K + 1);
            B->order = dmalloc<int32_t>(K);
            B->row_inst = dmalloc<int32_t>(m);
            B->dense = dmalloc<double>(dn[K]);
            B->dD = dmalloc<double>(m);
            B->refine = dmalloc<int32_t>(K);
            B->nref = dmalloc<int32_t>(2);
            check_cuda(cudaMemsetAsync(B->nref, 0, 2 * sizeof(int32_t), s), "memset");
            B->left_host = host_word();
            B->r = dmalloc<double>(m);
            B->ax = dmalloc<double>(m);
            B->nrp = dmalloc<int32_t>(m + 1);
            B->work = dmalloc<double>(m);
            B->solve_part = dmalloc<double>(2 * kFb * (m / kT + K + 1));
            check_cuda(cudaFuncSetAttribute(batch_ldlt_panel_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)panel_smem(kPanelT)),
                       "panel smem attribute");
            for (auto* k : {batch_ldlt_update_kernel<1>, batch_ldlt_update_kernel<2>})
                check_cuda(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kUpdSmem),
                           "update smem attribute");
            B->ref_iter = dmalloc<int32_t>(K);
            B->kkt = dmalloc<double>(4 * K);
            B->kkt_ref = dmalloc<double>(4 * K);
            check_cuda(cudaMemsetAsync(B->ref_iter, 0xff, sizeof(int32_t) * K, s), "memset");  // -1
            check_cuda(cudaMemsetAsync(B->kkt, 0, sizeof(double) * 4 * K, s), "memset");
            check_cuda(cudaMemsetAsync(B->kkt_ref, 0, sizeof(double) * 4 * K, s), "memset");
            check_cuda(cudaMemcpy(B->row_off, row_off_host, sizeof(int64_t) * (K + 1), cudaMemcpyHostToDevice), "H2D");
            check_cuda(cudaMemcpy(B->col_off, col_off_host, sizeof(int64_t) * (K + 1), cudaMemcpyHostToDevice), "H2D");
            check_cuda(cudaMemcpy(B->dn_off, dn.data(), sizeof(int64_t) * (K + 1), cudaMemcpyHostToDevice), "H2D");
            check_cuda(cudaMemcpy(B->order, order.data(), sizeof(int32_t) * K, cudaMemcpyHostToDevice), "H2D");
            launch_next(row_inst_kernel, (unsigned)K, 256, 0, s, K, B->row_off, B->row_inst);
            launched("row_inst_kernel");
            launch_next(narrow_rp_kernel, (unsigned)((m + 1 + 255) / 256), 256, 0, s, m + 1, P->rp, B->nrp);
            launched("narrow_rp_kernel");
            make_tile_table(B->nrp, m, P->nnz, &B->ntiles, &B->tile_row, &B->tile_nz, &B->carry_row, &B->carry_val,
                            &B->head_row, &B->head_val, &B->short_heads, s);
            // level schedule (instances in decreasing size: the ones with a block
            // at step s form a prefix of `order`)
            B->mmax = row_off_host[order[0] + 1] - row_off_host[order[0]];
            B->nsteps = (B->mmax + kFb - 1) / kFb;
            B->tile_off_h.assign(1, 0);
            B->chunk_off_h.assign(1, 0);
            std::vector<int64_t> tiles;
            std::vector<Chunk> chunks;
            for (int64_t st = 0; st < B->nsteps; ++st) {
                int32_t cnt = 0;
                int64_t acc = 0;
                for (int64_t b = 0; b < K; ++b) {
                    const int64_t mi = row_off_host[order[b] + 1] - row_off_host[order[b]];
                    if (mi <= st * kFb) break;
                    const int64_t rest = mi - std::min<int64_t>(mi, (st + 1) * kFb);
                    acc += update_tiles((rest + kFb - 1) / kFb, st % 2 == 0);
                    tiles.push_back(acc);
                    for (int32_t c = 0; c * kT < rest; ++c) chunks.push_back(Chunk{order[b], c});
                    ++cnt;
                }
                B->step_cnt.push_back(cnt);
                B->step_tiles_h.push_back(acc);
                B->tile_off_h.push_back((int64_t)tiles.size());
                B->chunk_off_h.push_back((int64_t)chunks.size());
            }
            // the solve's clusters, largest instances first. An instance gets
            // the CTAs that leave each of them at most `per` chunks of rows
            // below the first block, per as small as keeps the batch within
            // five CTAs per SM: few instances are split for latency, many
            // run side by side (one solve of 384 LPs of m 50-2000: per = 1, 2,
            // 4, 8 give 864, 568, 727, 951 us)
            auto group = [](int64_t mi, int64_t per) {
                const int64_t ch = (std::max<int64_t>(mi - kFb, 0) + kT - 1) / kT;
                int g = 1;
                while (g < kSolveCluster && ch > per * g) g *= 2;
                return g;
            };
            int64_t per = 1;
            for (;; per *= 2) {
                int64_t total = 0;
                for (int64_t i = 0; i < K; ++i) total += group(row_off_host[i + 1] - row_off_host[i], per);
                if (per == 8 || total <= 5 * (int64_t)ctx().sm_count) break;
            }
            std::vector<InstInfo> info(K);
            std::vector<SolveSlot> slots;
            int64_t alone_m = 1;
            for (int64_t b = 0; b < K; ++b) {
                const int32_t i = order[b];
                const int64_t mi = row_off_host[i + 1] - row_off_host[i];
                info[i] = InstInfo{row_off_host[i], dn[i], (int32_t)mi, {0, 0, 0}};
                const int size = group(mi, per);
                if (size == 1) alone_m = std::max(alone_m, mi);
                if (!slots.empty() && slots.back().size != size)
                    while (slots.size() % kSolveCluster)
                        slots.push_back(SolveSlot{-1, 0, 1, slots.back().steps});
                const int32_t steps = size == 1 ? 0
                                      : slots.size() % kSolveCluster ? slots.back().steps
                                                                     : (int32_t)((mi + kFb - 1) / kFb);
                for (int32_t r = 0; r < size; ++r) slots.push_back(SolveSlot{i, r, size, steps});
            }
            while (slots.size() % kSolveCluster) slots.push_back(SolveSlot{-1, 0, 1, slots.back().steps});
            B->nslots = (int64_t)slots.size();
            B->solve_smem = sizeof(double) * (2 * kFb * kSolveP + alone_m);  // alone_m <= 8 kT + kFb
            check_cuda(cudaFuncSetAttribute(batch_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)sizeof(double) * (2 * kFb * kSolveP + 8 * kT + kFb)),
                       "solve smem attribute");
            auto upload = [&](auto*& dst, const auto& src) {
                using T = std::remove_reference_t<decltype(*dst)>;
                dst = dmalloc<T>(src.size());
                if (!src.empty())
                    check_cuda(cudaMemcpy(dst, src.data(), sizeof(T) * src.size(), cudaMemcpyHostToDevice), "H2D schedule");
            };
            upload(B->step_tiles, tiles);
            upload(B->chunks, chunks);
            upload(B->info, info);
            upload(B->slots, slots);
            check_cuda(cudaStreamSynchronize(s), "batch create sync");
        } catch (...) {
            free_batch(B);
            throw;
        }
        *out = B;
    });
}

int hn_batch_destroy(hn_batch* B) {
    return guard("hn_batch_destroy", [&] {
        if (!B) return;
        require_init();
        cudaDeviceSynchronize();
        free_batch(B);
    });
}

int hn_batch_residuals(hn_batch* B, const hn_csr* M, const double* x, const double* lam, const double* z,
                       const double* b, const double* c, double* mx, double* rp, double* rd, double* D, double* Drd,
                       double* scal, int32_t* status, int32_t* iters, int iter, double tol, double ctol,
                       void* stream) {
    return guard("hn_batch_residuals", [&] {
        require_init();
        if (!B || !M || !M->has_t) fail(HN_ERR_INVALID_ARG, "bad arguments");
        cudaStream_t s = as_stream(stream);
        spmv_launch2(spmv_mat(M, 0), x, EpiResidual{b, mx, rp}, spmv_mat(M, 1), lam, EpiDualResidual{z, c, rd}, s);
        launch_next(batch_prep_kernel, (unsigned)B->K, kT, 0, s, B->row_off, B->col_off, x, z, rd, rp, D, Drd, scal,
                    status, iters, iter, tol, ctol, kkt_args(B, lam, b, c));
        launched("batch_prep_kernel");
    });
}

int hn_batch_set_kkt(hn_batch* B, const double* ru, const double* cu, const double* offset, double kkt_tol,
                     int extra_iterations) {
    return guard("hn_batch_set_kkt", [&] {
        require_init();
        if (!B || (ru == nullptr) != (cu == nullptr) || (ru && !offset) || extra_iterations < 0)
            fail(HN_ERR_INVALID_ARG, "bad arguments");
        if (kkt_tol > 0.0 && !ru) fail(HN_ERR_INVALID_ARG, "tightening needs the unscale factors");
        B->ru = ru;
        B->cu = cu;
        B->offset = offset;
        B->kkt_tol = kkt_tol > 0.0 ? kkt_tol : 0.0;
        B->kkt_extra = extra_iterations;
        if (B->kkt_tol > 0.0 && !B->xb) {
            B->xb = dmalloc<double>(B->n);
            B->zb = dmalloc<double>(B->n);
            B->lb = dmalloc<double>(B->m);
        }
        check_cuda(cudaMemset(B->ref_iter, 0xff, sizeof(int32_t) * B->K), "memset");
        check_cuda(cudaMemset(B->kkt, 0, sizeof(double) * 4 * B->K), "memset");
        check_cuda(cudaMemset(B->kkt_ref, 0, sizeof(double) * 4 * B->K), "memset");
    });
}

int hn_batch_kkt(const hn_batch* B, double* kkt_host, int32_t* ref_iter_host) {
    return guard("hn_batch_kkt", [&] {
        require_init();
        if (!B) fail(HN_ERR_INVALID_ARG, "null batch");
        check_cuda(cudaDeviceSynchronize(), "sync");
        if (kkt_host)
            check_cuda(cudaMemcpy(kkt_host, B->kkt, sizeof(double) * 4 * B->K, cudaMemcpyDeviceToHost), "D2H kkt");
        if (ref_iter_host)
            check_cuda(cudaMemcpy(ref_iter_host, B->ref_iter, sizeof(int32_t) * B->K, cudaMemcpyDeviceToHost),
                       "D2H ref_iter");
    });
}

int hn_batch_finish(hn_batch* B, double* x, double* z, double* lam, int32_t* status, int32_t* iters, void* stream) {
    return guard("hn_batch_finish", [&] {
        require_init();
        if (!B || !x || !z || !lam || !status || !iters) fail(HN_ERR_INVALID_ARG, "bad arguments");
        cudaStream_t s = as_stream(stream);
        launch_next(batch_finish_kernel, (unsigned)B->K, kT, 0, s, B->row_off, B->col_off, x, z, lam, status, iters,
                    kkt_args(B, lam, nullptr, nullptr));
        launched("batch_finish_kernel");
    });
}

int hn_batch_factor(hn_batch* B, const double* D, double reg, double singular_tol, double* nval,
                    const int32_t* status, void* stream) {
    return guard("hn_batch_factor", [&] {
        require_init();
        if (!B || !D || !nval || !status) fail(HN_ERR_INVALID_ARG, "bad arguments");
        cudaStream_t s = as_stream(stream);
        ada_numeric_unregularised(B->P, D, nval, s);
        launch_next(batch_reg_kernel, (unsigned)B->K, kT, 0, s, B->row_off, B->P->diag_pos, reg, status, nval);
        launched("batch_reg_kernel");
        launch_next(batch_dense_kernel, (unsigned)((B->m * 32 + 255) / 256), 256, 0, s, B->m, B->row_off, B->row_inst,
                    B->dn_off, status, B->P->rp, B->P->ci, nval, B->dense);
        launched("batch_dense_kernel");
        // steps in pairs: after an even step only the next block column is
        // brought up to date, after an odd one the rest, by both panels at once
        for (int64_t st = 0; st < B->nsteps; ++st) {
            const int cnt = B->step_cnt[st];
            const int64_t nb = B->mmax - st * kFb;  // the largest block's rows
            auto* diag = nb <= 16   ? batch_ldlt_diag_kernel<16>
                         : nb <= 32 ? batch_ldlt_diag_kernel<32>
                         : nb <= 48 ? batch_ldlt_diag_kernel<48>
                                    : batch_ldlt_diag_kernel<64>;
            launch_next(diag, cnt, (unsigned)std::min<int64_t>((nb + 15) / 16 * 64, 4 * kFb), 0, s, (int)st, B->info, B->order, status,
                        B->dense, B->dD, singular_tol);
            launched("batch_ldlt_diag_kernel");
            const int64_t nc = B->chunk_off_h[st + 1] - B->chunk_off_h[st];
            if (nc == 0) continue;
            if (nc <= kPanelWide)
                launch_next(batch_ldlt_panel_kernel<4>, (unsigned)(nc * (kT / (kPanelT / 4))), kPanelT,
                            panel_smem(kPanelT / 4), s, (int)st, B->chunks + B->chunk_off_h[st], B->info, status,
                            B->dense, B->dD);
            else
                launch_next(batch_ldlt_panel_kernel<1>, (unsigned)(nc * (kT / kPanelT)), kPanelT, panel_smem(kPanelT),
                            s, (int)st, B->chunks + B->chunk_off_h[st], B->info, status, B->dense, B->dD);
            launched("batch_ldlt_panel_kernel");
            const int64_t nt = B->step_tiles_h[st];
            const unsigned grid = (unsigned)std::min<int64_t>(nt, 2 * (int64_t)ctx().sm_count);
            const int kt = (int)(st + 1) * kFb;
            const int64_t* tiles = B->step_tiles + B->tile_off_h[st];
            if (st % 2 == 0)
                launch_next(batch_ldlt_update_kernel<1>, grid, kUpdT, kUpdSmem, s, kt - kFb, kt, 1, cnt, nt, tiles,
                            B->info, B->order, status, B->dense, B->dD);
            else
                launch_next(batch_ldlt_update_kernel<2>, grid, kUpdT, kUpdSmem, s, kt - 2 * kFb, kt, 0, cnt, nt,
                            tiles, B->info, B->order, status, B->dense, B->dD);
            launched("batch_ldlt_update_kernel");
        }
    });
}

int hn_batch_solve(hn_batch* B, const double* nval, const double* rhs, double* x, const int32_t* status,
                   void* stream) {
    return guard("hn_batch_solve", [&] {
        require_init();
        if (!B || !nval || !rhs || !x || !status) fail(HN_ERR_INVALID_ARG, "bad arguments");
        cudaStream_t s = as_stream(stream);
        launch_next(batch_refine_start_kernel, (unsigned)B->K, kT, 0, s, B->row_off, status, rhs, B->refine, x);
        launched("batch_refine_start_kernel");
        solve_all(B, status, nullptr, x, s);
        const SpmvMat N = n_mat(B, nval);
        for (int sweep = 0; sweep < 5; ++sweep) {
            spmv_launch(N, x, EpiAxpby{1.0, 0.0, B->ax}, s);
            launch_next(batch_refine_check_kernel, (unsigned)B->K, kT, 0, s, B->row_off, status, rhs, B->ax, B->r,
                        B->refine, B->nref, B->left_host);
            launched("batch_refine_check_kernel");
            check_cuda(cudaStreamSynchronize(s), "refine sync");
            if (*static_cast<volatile int32_t*>(B->left_host) == 0) break;
            solve_all(B, status, B->refine, B->r, s);
            launch_next(batch_axpy_masked_kernel, (unsigned)((B->m + 255) / 256), 256, 0, s, B->m, B->row_inst,
                        status, B->refine, B->r, x);
            launched("batch_axpy_masked_kernel");
        }
    });
}

int hn_batch_quotients(int64_t n, const double* a, const double* d, double* q, void* stream) {
    return guard("hn_batch_quotients", [&] {
        require_init();
        if (n < 0 || (n && (!a || !d || !q))) fail(HN_ERR_INVALID_ARG, "bad arguments");
        if (n == 0) return;
        launch_next(quotients_kernel, (unsigned)((n + 255) / 256), 256, 0, as_stream(stream), n, a, d, q);
        launched("quotients_kernel");
    });
}

int hn_batch_steps(hn_batch* B, const double* x, const double* dx, const double* z, const double* dz,
                   const double* dlam, double* scal, int32_t* status, void* stream) {
    return guard("hn_batch_steps", [&] {
        require_init();
        if (!B) fail(HN_ERR_INVALID_ARG, "null batch");
        cudaStream_t s = as_stream(stream);
        launch_next(batch_steps_kernel, (unsigned)B->K, kT, 0, s, B->row_off, B->col_off, x, dx, z, dz, dlam, scal,
                    status);
        launched("batch_steps_kernel");
    });
}

int hn_batch_corrector(hn_batch* B, const hn_csr* M, const double* x, const double* dx, const double* z,
                       const double* dz, const double* rhs_pred, double* zs, double* rhs, double* scal,
                       const int32_t* status, void* stream) {
    return guard("hn_batch_corrector", [&] {
        require_init();
        if (!B || !M) fail(HN_ERR_INVALID_ARG, "bad arguments");
        cudaStream_t s = as_stream(stream);
        launch_next(batch_corr_kernel, (unsigned)B->K, kT, 0, s, B->col_off, x, dx, z, dz, scal, status, zs);
        launched("batch_corr_kernel");
        spmv_launch(spmv_mat(M, 0), zs, EpiCorrRhs{rhs_pred, rhs}, s);
    });
}

int hn_batch_update(hn_batch* B, double* x, const double* dx, double* z, const double* dz, double* lam,
                    const double* dlam, const double* scal, int32_t* status, int32_t* iters, int iter,
                    void* stream) {
    return guard("hn_batch_update", [&] {
        require_init();
        if (!B) fail(HN_ERR_INVALID_ARG, "null batch");
        cudaStream_t s = as_stream(stream);
        launch_next(batch_update_kernel, (unsigned)B->K, kT, 0, s, B->row_off, B->col_off, x, dx, z, dz, lam, dlam,
                    scal, status, iters, iter);
        launched("batch_update_kernel");
    });
}

}  // extern "C"
