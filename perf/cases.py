"""The work a user of this library has it do, as measurable cases.

Each case goes through the public entry points (hnb200, gnn and the C ABI they
load): sparse products, the normal-equation assembly, the interior-point
iteration of one LP and of a batch, a whole batched solve, simplex pricing,
the set-up of a new LP and one training step of the warm-start network.
Sizes are those of bench.py, lpgen.py and the tests (m from 200 to 200,000
rows, n = 2.5 m columns, 6 or 8 nonzeros per column or Zipf(1.5) column
counts on [1, 2000]), and draw() spreads over the same ranges.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "indigenous-cpu-gpu-optimization-engine-for-indian-industry_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)
import gnn  # noqa: E402
import hnb200 as hn  # noqa: E402
import lpgen  # noqa: E402

F64 = torch.float64
REG = 1e-8  # the IPM's default regularisation of the normal equations
ZIPF_MAX = 2000


def listed():
    return [
        # y = A x and t = A^T lam of a small LP: latency of the two products
        {"name": "spmv_small", "kind": "spmv", "m": 200, "n": 500, "k": 8, "nnz": 0},
        # the same on the large LP whose sparse step bench.py times (A x - b, then A^T lam)
        {"name": "spmv_5m", "kind": "spmv", "m": 200_000, "n": 500_000, "k": 0, "nnz": 5_000_000},
        # and on the LP with the unscaled Zipf law, the largest product
        {"name": "spmv_17m", "kind": "spmv", "m": 200_000, "n": 500_000, "k": 0, "nnz": 17_000_000},
        # C = A B with a block of right-hand sides (the compute backend's spmm)
        {"name": "spmm_32", "kind": "spmm", "m": 20_000, "n": 50_000, "k": 8, "nnz": 0, "cols": 32, "trans": 0},
        # N = A D A^T + dyn_reg I on the large LP's structure at half its rows, every IPM iteration's assembly
        {"name": "ada_large", "kind": "ada", "m": 100_000, "n": 250_000, "k": 0, "nnz": 2_500_000},
        # the device work of one Mehrotra iteration of the m = 2,000 LP, the plain solver's loop around its factorisation
        {"name": "ipm_step_2k", "kind": "ipm", "m": 2000, "n": 5000, "k": 8, "nnz": 0},
        # one lockstep iteration of a batch of small LPs (branch-and-bound nodes, many small models)
        {"name": "batch_iter_small", "kind": "batch", "count": 48, "lo": 50, "hi": 300, "k": 6},
        # the same for the batch configuration: sizes log-uniform in [50, 2000]
        {"name": "batch_iter_2k", "kind": "batch", "count": 384, "lo": 50, "hi": 2000, "k": 6},
        # a whole batched solve, host LPs in and solutions out
        {"name": "lp_batch", "kind": "solve", "count": 64, "lo": 50, "hi": 400, "k": 6},
        # one revised-simplex pricing round on the large LP with partial pricing of 16 candidates
        {"name": "price_500k", "kind": "price", "m": 200_000, "n": 500_000, "k": 0, "nnz": 5_000_000, "cand": 16},
        # a new model: coefficient triplets to the device, pattern of the normal matrix, first assembly
        {"name": "setup_20k", "kind": "setup", "m": 20_000, "n": 50_000, "k": 8, "nnz": 0},
        # one training step (forward and backward) of the warm-start network on a batch of LPs
        {"name": "gnn_step", "kind": "gnn", "count": 24, "lo": 500, "hi": 4000, "k": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, lo, hi, nnz_max):
    """An LP shape: m rows over a logarithmic range, about 2.5 m columns, a
    uniform or a Zipf column law."""
    m = _log(rng, lo, hi)
    n = int(m * rng.uniform(1.5, 2.5)) + rng.randrange(2)
    if rng.random() < 0.5:
        k = rng.randint(4, 10)
        if k * n <= nnz_max:
            return {"m": m, "n": n, "k": k, "nnz": 0}
    return {"m": m, "n": n, "k": 0, "nnz": min(nnz_max, int(n * rng.uniform(4.0, 10.0)))}


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmm", "ada", "ipm", "batch", "batch", "solve", "price", "setup", "gnn"])
    if kind == "spmv":
        return {"kind": kind, **_shape(rng, 200, 200_000, 5_000_000)}
    if kind == "spmm":
        return {"kind": kind, **_shape(rng, 200, 20_000, 400_000), "cols": rng.choice([1, 3, 8, 17, 32]),
                "trans": rng.randrange(2)}
    if kind == "ada":
        return {"kind": kind, **_shape(rng, 2000, 80_000, 1_600_000)}
    if kind == "ipm":
        return {"kind": kind, **_shape(rng, 200, 20_000, 300_000)}
    if kind == "batch":
        hi = _log(rng, 200, 1500)
        return {"kind": kind, "count": _log(rng, 8, 200), "lo": 50, "hi": hi, "k": rng.randint(4, 8)}
    if kind == "solve":
        return {"kind": kind, "count": _log(rng, 8, 60), "lo": 50, "hi": _log(rng, 100, 380), "k": rng.randint(5, 7)}
    if kind == "price":
        return {"kind": kind, **_shape(rng, 2000, 180_000, 4_500_000), "cand": rng.choice([1, 4, 8, 16])}
    if kind == "setup":
        return {"kind": kind, **_shape(rng, 500, 18_000, 150_000)}
    return {"kind": kind, "count": rng.randint(2, 20), "lo": 500, "hi": _log(rng, 1000, 3800), "k": rng.randint(5, 8)}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, size, lo, hi):
    return torch.rand(size, generator=g, dtype=F64, device="cuda") * (hi - lo) + lo


def _zipf_counts(g, n, target):
    """Zipf(1.5) column counts on [1, 2000], rescaled towards `target` entries."""
    w = torch.arange(1, ZIPF_MAX + 1, dtype=F64, device="cuda") ** -1.5
    cdf = torch.cumsum(w, 0) / w.sum()
    c = torch.searchsorted(cdf, torch.rand(n, generator=g, dtype=F64, device="cuda")) + 1
    c = c.clamp(max=ZIPF_MAX)
    return torch.round(c.to(F64) * (target / float(c.sum()))).to(torch.int64).clamp(1, ZIPF_MAX)


def _matrix(case, g, which=0):
    """The scaled constraint matrix the IPM iterates on (rows, then columns
    divided by their largest entry), as device triplets in row order. Where
    its entries lie follows from the case (and `which` of a batch), their
    values from `g`."""
    m, n = case["m"], case["n"]
    gs = _gen(31 * m + n + 7919 * which)
    if case["nnz"]:
        cnt = _zipf_counts(gs, n, case["nnz"]).clamp(max=m // 2)
    else:
        cnt = torch.full((n,), case["k"], dtype=torch.int64, device="cuda")
    cols = torch.repeat_interleave(torch.arange(n, device="cuda"), cnt)
    rows = torch.randint(0, m, (cols.numel(),), generator=gs, device="cuda")
    key = torch.unique(rows * n + cols)
    rows, cols = key // n, key % n
    val = _uniform(g, key.numel(), 0.1, 1.0)
    val = torch.where(torch.rand(key.numel(), generator=g, device="cuda") < 0.5, -val, val)
    rmax = torch.zeros(m, dtype=F64, device="cuda").scatter_reduce_(0, rows, val.abs(), "amax")
    val = val / rmax[rows]
    cmax = torch.zeros(n, dtype=F64, device="cuda").scatter_reduce_(0, cols, val.abs(), "amax")
    val = val / cmax[cols]
    return rows, cols, val


def _row_ptr(rows, m):
    rp = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0)
    return rp


def _csr(case, g):
    rows, cols, val = _matrix(case, g)
    rp = _row_ptr(rows, case["m"])
    A = hn.Csr(case["m"], case["n"], rp.cpu().numpy(), cols.cpu().numpy(), val.cpu().numpy())
    return A, (rows, cols, val)


def _mul(tri, x, m):
    """A x in 64 bits from the triplets."""
    rows, cols, val = tri
    return torch.zeros((m,) + x.shape[1:], dtype=F64, device="cuda").index_add_(
        0, rows, (val.reshape(-1, *[1] * (x.dim() - 1))) * x[cols])


def _tmul(tri, y, n):
    rows, cols, val = tri
    return _mul((cols, rows, val), y, n)


def _point(g, m, n):
    """An interior point in mid-solve: some variables near their bound (x
    small, z not), the others basic."""
    e = torch.randn(n, generator=g, dtype=F64, device="cuda")
    x = torch.exp(1.5 * e) * _uniform(g, n, 0.5, 2.0)
    z = torch.exp(-1.5 * e) * _uniform(g, n, 0.5, 2.0)
    lam = torch.randn(m, generator=g, dtype=F64, device="cuda")
    return x, z, lam


def _new(*size):
    return torch.empty(size, dtype=F64, device="cuda")


def _batch_sizes(case):
    return lpgen.batch_sizes(case["count"], case["lo"], case["hi"], 2000).tolist()


def _lps(case, seed):
    return [lpgen.lp_uniform(m, (5 * m) // 2, case["k"], seed * 1000 + i)
            for i, m in enumerate(_batch_sizes(case))]


def _packed(case, g):
    """The batch's matrices, packed block-diagonally."""
    ms = _batch_sizes(case)
    ns = [(5 * m) // 2 for m in ms]
    ro, co = np.cumsum([0] + ms), np.cumsum([0] + ns)
    rows, cols, vals = [], [], []
    for i, (m, n) in enumerate(zip(ms, ns)):
        r, c, v = _matrix({"m": m, "n": n, "k": case["k"], "nnz": 0}, g, i)
        rows.append(r + int(ro[i]))
        cols.append(c + int(co[i]))
        vals.append(v)
    return ro.astype(np.int64), co.astype(np.int64), (torch.cat(rows), torch.cat(cols), torch.cat(vals))


class _Batch:
    """An hn_batch handle with the matrix and pattern it works on."""

    def __init__(self, ro, co, tri):
        m, n = int(ro[-1]), int(co[-1])
        rp = _row_ptr(tri[0], m)
        self.A = hn.Csr(m, n, rp.cpu().numpy(), tri[1].cpu().numpy(), tri[2].cpu().numpy())
        self.P = hn.Pattern(self.A)
        self.h = C.c_void_p()
        p = C.POINTER(C.c_int64)
        hn.check(hn.load().hn_batch_create(len(ro) - 1, ro.ctypes.data_as(p), co.ctypes.data_as(p), self.P.h,
                                           C.byref(self.h)))

    def __del__(self):
        if self.h:
            hn.load().hn_batch_destroy(self.h)


def prepare(case, seed):
    hn.init(0)
    g, kind = _gen(seed), case["kind"]
    if kind == "solve":
        return {"kind": kind, "lps": _lps(case, seed)}
    if kind == "gnn":
        lps = _lps(case, seed)
        B = gnn.Batch(lps, [(lp["x0"], lp["y0"], lp["s0"]) for lp in lps])
        return {"kind": kind, "model": gnn.Model(seed=seed), "B": B}
    if kind == "batch":
        ro, co, tri = _packed(case, g)
        m, n, K = int(ro[-1]), int(co[-1]), case["count"]
        s = {"kind": kind, "B": _Batch(ro, co, tri), "K": K, "m": m, "n": n}
        s["x"], s["z"], s["lam"] = _point(g, m, n)
        s["b"] = _uniform(g, m, -4.0, 4.0)
        s["c"] = _uniform(g, n, 0.5, 4.0)
        for v in ("mx", "rp", "pred", "rhs", "dlam"):
            s[v] = _new(m)
        for v in ("rd", "D", "Drd", "dx", "dz", "zs"):
            s[v] = _new(n)
        s["nval"] = _new(s["B"].P.nnz)
        s["scal"] = torch.zeros(8 * K, dtype=F64, device="cuda")
        s["status"], s["iters"] = (torch.zeros(K, dtype=torch.int32, device="cuda") for _ in range(2))
        return s
    if kind == "setup":
        rows, cols, val = _matrix(case, g)
        order = torch.randperm(rows.numel(), generator=g, device="cuda")  # a file's order, not the matrix's
        return {"kind": kind, "m": case["m"], "n": case["n"], "rows": rows[order].cpu().numpy(),
                "cols": cols[order].cpu().numpy(), "val": val[order].cpu().numpy(),
                "D": torch.exp(torch.randn(case["n"], generator=g, dtype=F64, device="cuda"))}
    A, tri = _csr(case, g)
    m, n = case["m"], case["n"]
    s = {"kind": kind, "A": A, "m": m, "n": n}
    if kind == "spmv":
        s["x"], _, s["lam"] = _point(g, m, n)
        s["b"] = _uniform(g, m, -4.0, 4.0)
        s["y"], s["t"] = _new(m), _new(n)
    elif kind == "spmm":
        k, trans = case["cols"], case["trans"]
        s["k"], s["trans"] = k, trans
        s["X"] = torch.randn((m if trans else n, k), generator=g, dtype=F64, device="cuda")
        s["Y"] = _new(n if trans else m, k)
    elif kind == "ada":
        s["P"] = hn.Pattern(A)
        x, z, _ = _point(g, m, n)
        s["D"], s["nval"], s["dyn"] = x / z, _new(s["P"].nnz), _new(1)
    elif kind == "ipm":
        s["P"] = hn.Pattern(A)
        s["x"], s["z"], s["lam"] = _point(g, m, n)
        s["b"] = _uniform(g, m, -4.0, 4.0)
        s["c"] = _uniform(g, n, 0.5, 4.0)
        # the two solves belong to the host factorisation: their results are inputs here
        s["dlam1"], s["dlam2"] = (torch.randn(m, generator=g, dtype=F64, device="cuda") for _ in range(2))
        for v in ("mx", "rp", "pred", "rhs"):
            s[v] = _new(m)
        for v in ("rd", "D", "Drd", "dx1", "dz1", "dx", "dz", "zs"):
            s[v] = _new(n)
        s["nval"], s["dyn"] = _new(s["P"].nnz), _new(1)
        s["scal"] = torch.zeros(8, dtype=F64, device="cuda")
    elif kind == "price":
        s["k"] = case["cand"]
        s["yd"] = torch.randn(m, generator=g, dtype=F64, device="cuda")
        s["cost"] = torch.randn(n, generator=g, dtype=F64, device="cuda")
        s["u"] = torch.randn(m, generator=g, dtype=F64, device="cuda")
        s["nonbasis"] = torch.arange(n, dtype=torch.int32, device="cuda")
        s["nonbasis"][torch.randperm(n, generator=g, device="cuda")[:m]] = -1
        s["art"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
        s["w"] = _uniform(g, n, 1.0, 4.0)
        s["rc"], s["alpha"], s["colv"] = _new(n), _new(n), _new(case["cand"] * m)
        s["out"] = torch.zeros(case["cand"] + 1, dtype=torch.int64, device="cuda")
    return s


# ---------------------------------------------------------------- one pass
def _ptrs(s, names):
    return [s[v].data_ptr() for v in names.split()]


def _run_ipm(s):
    lib, A = hn.load(), s["A"].h
    ck = hn.check
    ck(lib.hn_ipm_residuals(A, *_ptrs(s, "x lam z b c mx rp rd D Drd scal"), None))
    s["P"].numeric(s["D"], REG, s["nval"], s["dyn"])
    ck(lib.hn_ipm_rhs(A, *_ptrs(s, "Drd rp mx pred"), None))
    ck(lib.hn_ipm_direction(A, *_ptrs(s, "dlam1 D rd x"), None, *_ptrs(s, "dx1 dz1"), None))
    ck(lib.hn_ipm_step_lengths(s["n"], s["m"], *_ptrs(s, "x dx1 z dz1 dlam1 scal"), None))
    ck(lib.hn_ipm_corrector(A, *_ptrs(s, "x dx1 z dz1 pred zs rhs scal"), None))
    ck(lib.hn_ipm_direction(A, *_ptrs(s, "dlam2 D rd x zs dx dz"), None))
    ck(lib.hn_ipm_step_lengths(s["n"], s["m"], *_ptrs(s, "x dx z dz dlam2 scal"), None))
    return {v: s[v] for v in ("mx", "rp", "rd", "D", "Drd", "nval", "dyn", "pred", "dx1", "dz1", "zs", "rhs", "dx",
                              "dz", "scal")}


def _run_batch(s):
    lib, B, A = hn.load(), s["B"].h, s["B"].A.h
    ck = hn.check
    ck(lib.hn_batch_residuals(B, A, *_ptrs(s, "x lam z b c mx rp rd D Drd scal status iters"), 0, 1e-8, 1e-8, None))
    ck(lib.hn_batch_factor(B, s["D"].data_ptr(), REG, 1e-12, *_ptrs(s, "nval status"), None))
    ck(lib.hn_ipm_rhs(A, *_ptrs(s, "Drd rp mx pred"), None))
    ck(lib.hn_batch_solve(B, *_ptrs(s, "nval pred dlam status"), None))
    ck(lib.hn_ipm_direction(A, *_ptrs(s, "dlam D rd x"), None, *_ptrs(s, "dx dz"), None))
    ck(lib.hn_batch_steps(B, *_ptrs(s, "x dx z dz dlam scal status"), None))
    ck(lib.hn_batch_corrector(B, A, *_ptrs(s, "x dx z dz pred zs rhs scal status"), None))
    ck(lib.hn_batch_solve(B, *_ptrs(s, "nval rhs dlam status"), None))
    ck(lib.hn_ipm_direction(A, *_ptrs(s, "dlam D rd x zs dx dz"), None))
    ck(lib.hn_batch_steps(B, *_ptrs(s, "x dx z dz dlam scal status"), None))
    return {v: s[v] for v in ("mx", "rp", "rd", "D", "nval", "pred", "zs", "rhs", "dlam", "dx", "dz", "scal",
                              "status")}


def _run_setup(s):
    A = hn.Csr.from_coo(s["m"], s["n"], s["rows"], s["cols"], s["val"])
    P = hn.Pattern(A)
    nval, dyn = _new(P.nnz), _new(1)
    P.numeric(s["D"], REG, nval, dyn)
    # the host factorisation's ordering reads the pattern
    rp = torch.empty(s["m"] + 1, dtype=torch.int64, device="cuda")
    ci = torch.empty(P.nnz, dtype=torch.int32, device="cuda")
    rpd, cid, _ = P.device_arrays()
    lib = hn.load()
    hn.check(lib.hn_memcpy_d2d(rp.data_ptr(), rpd, 8 * rp.numel(), None))
    hn.check(lib.hn_memcpy_d2d(ci.data_ptr(), cid, 4 * ci.numel(), None))
    P.close()
    A.close()
    return {"rp": rp, "ci": ci, "nval": nval, "dyn": dyn}


def run(state):
    s, kind = state, state["kind"]
    if kind == "spmv":
        s["A"].residual(s["x"], s["b"], s["y"])
        s["A"].spmv(s["lam"], s["t"], trans=1)
        return {"y": s["y"], "t": s["t"]}
    if kind == "spmm":
        s["A"].spmm(s["X"], s["k"], s["Y"], trans=s["trans"])
        return s["Y"]
    if kind == "ada":
        s["P"].numeric(s["D"], REG, s["nval"], s["dyn"])
        return {"nval": s["nval"], "dyn": s["dyn"]}
    if kind == "ipm":
        return _run_ipm(s)
    if kind == "batch":
        return _run_batch(s)
    if kind == "solve":
        r = hn.lp_solve_batch(s["lps"])
        return {v: r[v] for v in ("x", "y", "s", "objective", "status")}
    if kind == "price":
        hn.price_reduced_costs(s["A"], s["yd"], s["cost"], s["rc"])
        hn.price_devex_update(s["A"], s["u"], s["nonbasis"], s["w"], s["alpha"])
        hn.price_select(s["n"], s["rc"], s["w"], s["nonbasis"], s["art"], s["out"], k=s["k"])
        hn.price_columns(s["A"], s["out"][1:], s["colv"])
        return {v: s[v] for v in ("rc", "w", "alpha", "out", "colv")}
    if kind == "setup":
        return _run_setup(s)
    cache = gnn.forward(s["model"], s["B"])
    loss = gnn.backward(s["model"], s["B"], cache)
    return {"ov": cache["ov"], "oc": cache["oc"], "grad": s["model"].g, "loss": loss}


# ---------------------------------------------------------------- what a pass cannot do without
def _nnz(case):
    return case["nnz"] or case["k"] * case["n"]


def _terms(case):
    """Terms of A D A^T, the sum over columns of count^2 (their law's mean)."""
    if not case["nnz"]:
        return case["n"] * case["k"] ** 2
    k = np.arange(1, ZIPF_MAX + 1, dtype=np.float64)
    w = k ** -1.5 / np.sum(k ** -1.5)
    f = case["nnz"] / case["n"] / np.sum(w * k)
    return int(case["n"] * np.sum(w * np.maximum(1.0, f * k) ** 2))


def _slots(case):
    """Slots of N: its terms but for those that meet, and never above m^2."""
    m2 = float(case["m"]) ** 2
    return int(m2 * -math.expm1(-_terms(case) / m2)) + case["m"]


def _mean_power(case, p):
    lo, hi = float(case["lo"]), float(case["hi"])
    return (hi ** p - lo ** p) / (p * math.log(hi / lo)) if hi > lo else lo ** p


def work(case):
    kind = case["kind"]
    if kind in ("batch", "solve"):
        K, m1 = case["count"], _mean_power(case, 1)
        m2, m3 = _mean_power(case, 2), _mean_power(case, 3)
        nnz = 2.5 * m1 * case["k"]
        it = 1 if kind == "batch" else 15  # iterations a small LP takes at the least
        # L written once and read by the two sweeps of two solves, A and A^T by the products, N's terms
        by = K * (8 * m2 / 2 * 5 + 7 * 12 * nnz + 12 * min(m2, 2.5 * m1 * case["k"] ** 2) + 8 * 20 * 2.5 * m1)
        return {"bytes": int(it * by), "flops": int(it * K * (m3 / 3 + 4 * 2 * m2))}
    if kind == "gnn":
        m1 = _mean_power(case, 1) * case["count"]
        rows, nnz = 3.5 * m1, 2.5 * m1 * case["k"]
        act, layers = rows * gnn.H * 4, gnn.LAYERS
        # per layer: activations and aggregates written, read again by the backward, their gradients
        by = layers * (10 * act + 4 * 12 * nnz) + 6 * act
        fl = layers * (3 * 2 * rows * 2 * gnn.H * gnn.H + 4 * 2 * nnz * gnn.H) + 6 * rows * gnn.H * gnn.H
        return {"bytes": int(by), "flops": int(fl)}
    m, n, nnz = case["m"], case["n"], _nnz(case)
    mat = 12 * nnz
    if kind == "spmv":
        return {"bytes": 2 * mat + 4 * (m + n) + 8 * (2 * n + 4 * m), "flops": 4 * nnz}
    if kind == "spmm":
        return {"bytes": mat + 8 * case["cols"] * (m + n), "flops": 2 * nnz * case["cols"]}
    if kind == "ada":
        return {"bytes": mat + 8 * n + 12 * _slots(case) + 8 * m, "flops": 3 * _terms(case)}
    if kind == "ipm":
        return {"bytes": 6 * mat + 8 * (30 * n + 20 * m) + 12 * _slots(case), "flops": 12 * nnz + 3 * _terms(case)}
    if kind == "price":
        return {"bytes": 2 * mat + 8 * (6 * n + 2 * m) + 5 * n + 8 * case["cand"] * m, "flops": 4 * nnz}
    return {"bytes": 24 * nnz + 12 * nnz + 24 * _slots(case), "flops": 3 * _terms(case)}


# ---------------------------------------------------------------- the same in 64 bits, without the library
def _normal(tri, D, m, rows_per=4_000_000):
    """A D A^T's pattern (diagonal included) and values before dyn_reg, as
    sorted keys i * m + k."""
    rows, cols, val = tri
    order = torch.argsort(cols, stable=True)
    r, c, v = rows[order], cols[order], val[order]
    cnt = torch.bincount(c, minlength=D.numel())
    start = torch.cumsum(cnt, 0) - cnt
    keys, vals = [torch.arange(m, device="cuda") * (m + 1)], [torch.zeros(m, dtype=F64, device="cuda")]
    for a in range(0, r.numel(), rows_per):
        e = torch.arange(a, min(a + rows_per, r.numel()), device="cuda")
        reps = cnt[c[e]]
        left = torch.repeat_interleave(e, reps)
        inner = torch.arange(left.numel(), device="cuda") - torch.repeat_interleave(torch.cumsum(reps, 0) - reps, reps)
        right = start[c[left]] + inner
        keys.append(r[left] * m + r[right])
        vals.append(v[left] * v[right] * D[c[left]])
        del left, inner, right
    key, inv = torch.unique(torch.cat(keys), return_inverse=True)
    del keys
    out = torch.zeros(key.numel(), dtype=F64, device="cuda").index_add_(0, inv, torch.cat(vals))
    return key, out


def _regularise(key, val, m, lo=0):
    """dyn_reg = max(reg, 1e-12 max diagonal) on the diagonal."""
    d = torch.searchsorted(key, torch.arange(m, device="cuda") * (m + 1))
    dyn = max(REG, 1e-12 * float(val[d].max()))
    val[d] += dyn
    return dyn


def _clamped(x, z):
    D = x / z
    return torch.where((D >= 0) & (D <= 1e10), D, torch.full_like(D, 1e10))


def _max_step(v, d):
    r = torch.where(d < 0, -v / d, torch.ones_like(v))
    return min(1.0, 0.99 * min(1.0, float(r.min())))


def _sigma(mu_aff, mu):
    if not math.isfinite(mu_aff) or mu_aff < 0.0 or not mu > 0.0:
        return 0.5
    return min(0.9, max(0.1, (mu_aff / max(mu, 1e-300)) ** 3))


def _corrector(x, dx, z, dz, mu):
    ap, ad = _max_step(x, dx), _max_step(z, dz)
    mu_aff = float(((x + ap * dx) * (z + ad * dz)).sum()) / x.numel()
    sig = _sigma(mu_aff, mu)
    return mu_aff, sig, (sig * mu - dx * dz) / z


def _exact_ipm(case, seed):
    g = _gen(seed)
    tri = _matrix(case, g)
    m, n = case["m"], case["n"]
    x, z, lam = _point(g, m, n)
    b = _uniform(g, m, -4.0, 4.0)
    c = _uniform(g, n, 0.5, 4.0)
    dl1, dl2 = (torch.randn(m, generator=g, dtype=F64, device="cuda") for _ in range(2))
    o = {"mx": _mul(tri, x, m)}
    o["rp"] = o["mx"] - b
    o["rd"] = _tmul(tri, lam, n) + z - c
    o["D"] = _clamped(x, z)
    o["Drd"] = o["D"] * o["rd"]
    key, o["nval"] = _normal(tri, o["D"], m)
    o["dyn"] = torch.full((1,), _regularise(key, o["nval"], m), dtype=F64)
    o["pred"] = -o["rp"] - _mul(tri, o["Drd"], m) + o["mx"]
    u = _tmul(tri, dl1, n) + o["rd"]
    o["dx1"], o["dz1"] = o["D"] * u - x, -u
    mu = float((x * z).sum()) / n
    mu_aff, sig, o["zs"] = _corrector(x, o["dx1"], z, o["dz1"], mu)
    o["rhs"] = o["pred"] - _mul(tri, o["zs"], m)
    u = _tmul(tri, dl2, n) + o["rd"]
    o["dx"], o["dz"] = o["D"] * u - x + o["zs"], -u
    bad = 0.0  # the FLAGS slot: no entry is out of range
    o["scal"] = torch.tensor([float(o["rp"].abs().max()), float(o["rd"].abs().max()), mu, _max_step(x, o["dx"]),
                              _max_step(z, o["dz"]), mu_aff, sig, bad], dtype=F64)
    return o


def _exact_batch(case, seed):
    if case["count"] * _mean_power(case, 3) > 4e11:
        return None
    g = _gen(seed)
    ro, co, tri = _packed(case, g)
    m, n, K = int(ro[-1]), int(co[-1]), case["count"]
    x, z, lam = _point(g, m, n)
    b = _uniform(g, m, -4.0, 4.0)
    c = _uniform(g, n, 0.5, 4.0)
    o = {"mx": _mul(tri, x, m)}
    o["rp"] = o["mx"] - b
    o["rd"] = _tmul(tri, lam, n) + z - c
    D = o["D"] = _clamped(x, z)
    o["pred"] = -o["rp"] - _mul(tri, D * o["rd"], m) + o["mx"]
    key, o["nval"] = _normal(tri, D, m)
    facs, scal = [], torch.zeros(K, 8, dtype=F64)
    ki, kk = key // m, key % m
    cuts = torch.searchsorted(key, torch.as_tensor(ro, device="cuda") * m).tolist()
    for i in range(K):
        r0, r1 = int(ro[i]), int(ro[i + 1])
        a, e = cuts[i], cuts[i + 1]
        N = torch.zeros(r1 - r0, r1 - r0, dtype=F64, device="cuda")
        d = ki[a:e] == kk[a:e]
        o["nval"][a:e][d] += max(REG, 1e-12 * float(o["nval"][a:e][d].max()))
        N[ki[a:e] - r0, kk[a:e] - r0] = o["nval"][a:e]
        facs.append(torch.linalg.cholesky(N))

    def solve(rhs):
        return torch.cat([torch.cholesky_solve(rhs[int(ro[i]):int(ro[i + 1]), None], facs[i])[:, 0] for i in range(K)])

    dlam = solve(o["pred"])
    u = _tmul(tri, dlam, n) + o["rd"]
    dx, dz = D * u - x, -u
    o["zs"] = torch.empty_like(x)
    for i in range(K):
        q = slice(int(co[i]), int(co[i + 1]))
        mu = float((x[q] * z[q]).sum()) / (q.stop - q.start)
        mu_aff, sig, o["zs"][q] = _corrector(x[q], dx[q], z[q], dz[q], mu)
        scal[i, 2], scal[i, 5], scal[i, 6] = mu, mu_aff, sig
    o["rhs"] = o["pred"] - _mul(tri, o["zs"], m)
    o["dlam"] = solve(o["rhs"])
    u = _tmul(tri, o["dlam"], n) + o["rd"]
    o["dx"], o["dz"] = D * u - x + o["zs"], -u
    for i in range(K):
        q, p = slice(int(co[i]), int(co[i + 1])), slice(int(ro[i]), int(ro[i + 1]))
        scal[i, 0], scal[i, 1] = float(o["rp"][p].abs().max()), float(o["rd"][q].abs().max())
        scal[i, 3], scal[i, 4] = _max_step(x[q], o["dx"][q]), _max_step(z[q], o["dz"][q])
    o["scal"], o["status"] = scal.reshape(-1), None
    return o


def _exact_gnn(case, seed):
    lps = _lps(case, seed)
    rp, ci, m_off, n_off = gnn.pack(lps)
    m, n = int(m_off[-1]), int(n_off[-1])
    rows = torch.as_tensor(np.repeat(np.arange(m), np.diff(rp)), device="cuda")
    cols = torch.as_tensor(ci, device="cuda")
    vr, vc = (torch.as_tensor(np.concatenate(v), device="cuda") for v in zip(*(gnn.normalised_values(p) for p in lps)))
    F = [gnn.features(p) for p in lps]
    T = [gnn.targets(p["x0"], p["y0"], p["s0"]) for p in lps]
    Fv, Fc, Tv, Tc = (torch.as_tensor(np.concatenate(v), device="cuda").to(F64)
                      for v in (*zip(*F), *zip(*T)))
    off, size = gnn.param_offsets()
    w = torch.as_tensor(gnn.init_params(seed), device="cuda").to(F64).requires_grad_(True)

    def lin(x, name, relu=True):
        o, K = off[name]
        y = x @ w[o:o + K * gnn.H].reshape(K, gnn.H) + w[o + K * gnn.H:o + K * gnn.H + gnn.H]
        return torch.relu(y) if relu else y

    hv, hc = lin(Fv, "ev"), lin(Fc, "ec")
    for la in range(gnn.LAYERS):
        a = torch.zeros(m, gnn.H, dtype=F64, device="cuda").index_add(0, rows, vr[:, None] * hv[cols])
        hc = lin(torch.cat([hc, a], 1), f"c{la}")
        a = torch.zeros(n, gnn.H, dtype=F64, device="cuda").index_add(0, cols, vc[:, None] * hc[rows])
        hv = lin(torch.cat([hv, a], 1), f"v{la}")
    ov, oc = lin(hv, "hv", False), lin(hc, "hc", False)
    loss = ((ov[:, :2] - Tv) ** 2).sum() / n + ((oc[:, 0] - Tc[:, 0]) ** 2).sum() / m
    loss.backward()
    return {"ov": ov.detach(), "oc": oc.detach(), "grad": w.grad, "loss": float(loss.detach())}


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return None  # an optimum within its stopping tolerance has no such value
    if kind == "gnn":
        return _exact_gnn(case, seed)
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "ipm":
        return _exact_ipm(case, seed)
    g = _gen(seed)
    tri = _matrix(case, g)
    m, n = case["m"], case["n"]
    if kind == "spmv":
        x, _, lam = _point(g, m, n)
        b = _uniform(g, m, -4.0, 4.0)
        return {"y": _mul(tri, x, m) - b, "t": _tmul(tri, lam, n)}
    if kind == "spmm":
        X = torch.randn((m if case["trans"] else n, case["cols"]), generator=g, dtype=F64, device="cuda")
        return _tmul(tri, X, n) if case["trans"] else _mul(tri, X, m)
    if kind == "ada":
        x, z, _ = _point(g, m, n)
        key, val = _normal(tri, x / z, m)
        dyn = _regularise(key, val, m)
        return {"nval": val, "dyn": torch.full((1,), dyn, dtype=F64)}
    if kind == "setup":
        torch.randperm(tri[0].numel(), generator=g, device="cuda")
        D = torch.exp(torch.randn(n, generator=g, dtype=F64, device="cuda"))
        key, val = _normal(tri, D, m)
        dyn = _regularise(key, val, m)
        return {"rp": None, "ci": None, "nval": val, "dyn": torch.full((1,), dyn, dtype=F64)}
    # price
    yd = torch.randn(m, generator=g, dtype=F64, device="cuda")
    cost = torch.randn(n, generator=g, dtype=F64, device="cuda")
    u = torch.randn(m, generator=g, dtype=F64, device="cuda")
    nonb = torch.ones(n, dtype=torch.bool, device="cuda")
    nonb[torch.randperm(n, generator=g, device="cuda")[:m]] = False
    w = _uniform(g, n, 1.0, 4.0)
    rc, alpha = cost - _tmul(tri, yd, n), _tmul(tri, u, n)
    w = torch.where(nonb, torch.maximum(w, (alpha / alpha[nonb].abs().max()) ** 2), w)
    return {"rc": rc, "w": w, "alpha": alpha, "out": None, "colv": None}
