"""GPU: hn_batch_factor + hn_batch_solve against numpy on each instance's N.

Sizes sit on the edges of the kernels' blocks: 64-column steps and their
pairs, 128-row panel parts, 256-row chunks, and the row counts at which an
instance's solve goes from one CTA to two, four and eight. Values far outside
2^-400 .. 2^400 take the factorisation's dividing path.

Bar: forward error of a backward-stable factorisation, 50 m eps cond(N) in
the 2-norm (numpy's own included).
"""
import ctypes as C

import numpy as np
import pytest

import lpgen

pytestmark = pytest.mark.gpu


def solve_batch(hn, torch, ms, scale=1.0, masked=()):
    lps = [lpgen.lp_uniform(m, 3 * m, min(4, m), 50 + i) for i, m in enumerate(ms)]
    ro = np.cumsum([0] + list(ms)).astype(np.int64)
    co = np.cumsum([0] + [3 * m for m in ms]).astype(np.int64)
    rp = np.concatenate([[0]] + [lp["rp"][1:] + sum(len(p["ci"]) for p in lps[:i]) for i, lp in enumerate(lps)])
    ci = np.concatenate([lp["ci"] + co[i] for i, lp in enumerate(lps)])
    val = np.concatenate([lp["val"] for lp in lps])
    A = hn.Csr(int(ro[-1]), int(co[-1]), rp, ci, val, autotune=False)
    P = hn.Pattern(A)
    rng = np.random.default_rng(7)
    D, rhs = rng.uniform(0.5, 2.0, co[-1]) * scale, rng.standard_normal(ro[-1])
    dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
    nval = torch.empty(P.nnz, dtype=torch.float64, device="cuda")
    status = np.zeros(len(ms), np.int32)
    status[list(masked)] = 1
    Dd, rd, st, x = dev(D), dev(rhs), dev(status), torch.empty(int(ro[-1]), dtype=torch.float64, device="cuda")
    lib, h = hn.load(), C.c_void_p()
    p64 = C.POINTER(C.c_int64)
    hn.check(lib.hn_batch_create(len(ms), ro.ctypes.data_as(p64), co.ctypes.data_as(p64), P.h, C.byref(h)))
    try:
        hn.check(lib.hn_batch_factor(h, Dd.data_ptr(), 0.0, 1e-300, nval.data_ptr(), st.data_ptr(), None))
        hn.check(lib.hn_batch_solve(h, nval.data_ptr(), rd.data_ptr(), x.data_ptr(), st.data_ptr(), None))
        torch.cuda.synchronize()
    finally:
        hn.check(lib.hn_batch_destroy(h))
    return lps, ro, co, D, rhs, x.cpu().numpy()


def check(i, lps, ro, co, D, rhs, x, scale):
    lp = lps[i]
    m, n = lp["m"], lp["n"]
    A = np.zeros((m, n))
    A[np.repeat(np.arange(m), np.diff(lp["rp"])), lp["ci"]] = lp["val"]
    N = (A * (D[co[i]:co[i + 1]] / scale)) @ A.T
    N[np.diag_indices(m)] += 1e-12 * N.diagonal().max()
    ref = np.linalg.solve(N, rhs[ro[i]:ro[i + 1]])
    got = x[ro[i]:ro[i + 1]] * scale
    tol = 50 * m * np.finfo(float).eps * np.linalg.cond(N)
    assert np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref), (m, np.linalg.norm(got - ref), tol)


@pytest.mark.parametrize("scale", [1.0, 1e-140, 1e130])
def test_block_edges(hn, torch_cuda, scale):
    ms = [1, 2, 63, 64, 65, 127, 128, 129, 191, 192, 193, 256, 257, 319, 320, 321]
    r = solve_batch(hn, torch_cuda, ms, scale)
    for i in range(len(ms)):
        check(i, *r, scale)


@pytest.mark.parametrize("ms", [[1100, 1089, 1088, 833, 832, 577, 576, 449, 322], [1345], [400, 1, 400]])
def test_solve_groups_and_masks(hn, torch_cuda, ms):
    """Few instances: several CTAs each; a masked instance keeps its right-hand side."""
    masked = [1] if len(ms) > 1 else []
    r = solve_batch(hn, torch_cuda, ms, masked=masked)
    for i in range(len(ms)):
        if i in masked:
            assert np.array_equal(r[5][r[1][i]:r[1][i + 1]], r[4][r[1][i]:r[1][i + 1]])
        else:
            check(i, *r, 1.0)


def test_many_instances_one_cta_each(hn, torch_cuda):
    """Enough instances that those with several row chunks still get one CTA."""
    ms = [330, 70] * 400 + [900]
    r = solve_batch(hn, torch_cuda, ms)
    for i in list(range(0, 800, 97)) + [800]:
        check(i, *r, 1.0)


@pytest.mark.parametrize("scale", [1.0, 1e-140, 1e130])
def test_many_panel_rows(hn, torch_cuda, scale):
    """Enough rows below the first block for a panel row per lane (few: four lanes per row)."""
    ms = [65, 128, 193, 257, 321] * 24
    r = solve_batch(hn, torch_cuda, ms, scale)
    for i in [0, 1, 2, 3, 4, 61, 117, 118, 119]:
        check(i, *r, scale)


def test_many_handles_at_once(hn, torch_cuda):
    """More handles than one slab of their host words has room for, solved in
    turn; their words are used again."""
    import threading

    lib, p64, n = hn.load(), C.POINTER(C.c_int64), 1100
    A = hn.Csr(3, 3, [0, 1, 2, 4], [0, 1, 1, 2], [2.0, 1.0, 1.0, 1.0])
    P = hn.Pattern(A)
    ro = np.array([0, 3], np.int64)
    dev = lambda a: torch_cuda.as_tensor(np.asarray(a), device="cuda")  # noqa: E731
    D, rhs, st = dev(np.ones(3)), dev([1.0, -2.0, 3.0]), dev(np.zeros(1, np.int32))
    N = np.array([[4.0, 0, 0], [0, 1, 1], [0, 1, 2]])
    N[np.diag_indices(3)] += 4e-12
    want = np.linalg.solve(N, [1.0, -2.0, 3.0])

    def create():
        h = C.c_void_p()
        hn.check(lib.hn_batch_create(1, ro.ctypes.data_as(p64), ro.ctypes.data_as(p64), P.h, C.byref(h)))
        return h

    def solve(h):
        nval, x = torch_cuda.empty(P.nnz, dtype=torch_cuda.float64, device="cuda"), torch_cuda.empty_like(rhs)
        hn.check(lib.hn_batch_factor(h, D.data_ptr(), 0.0, 1e-300, nval.data_ptr(), st.data_ptr(), None))
        hn.check(lib.hn_batch_solve(h, nval.data_ptr(), rhs.data_ptr(), x.data_ptr(), st.data_ptr(), None))
        torch_cuda.cuda.synchronize()
        assert np.allclose(x.cpu().numpy(), want, rtol=1e-12, atol=0)

    hs = [create() for _ in range(n)]
    for h in hs[::97] + hs[-1:]:
        solve(h)
    for h in hs[: n // 2]:
        hn.check(lib.hn_batch_destroy(h))
    hs = [create() for _ in range(n // 2)] + hs[n // 2:]
    errors = []

    def work(part):
        try:
            for h in part:
                hn.check(lib.hn_batch_destroy(h))
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    solve(hs[0])
    ts = [threading.Thread(target=work, args=(hs[t::4],)) for t in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors, errors
    h = create()
    solve(h)
    hn.check(lib.hn_batch_destroy(h))


@pytest.mark.parametrize("m", [2112, 2113, 2369, 4200])
def test_several_chunks_per_cta(hn, torch_cuda, m):
    """One instance on a group of eight CTAs with one chunk of rows each or several, the same bits every time."""
    r = solve_batch(hn, torch_cuda, [m])
    check(0, *r, 1.0)
    for _ in range(3):
        assert np.array_equal(solve_batch(hn, torch_cuda, [m])[5], r[5])


def test_groups_of_two_and_four(hn, torch_cuda):
    """Enough instances for up to two chunks of rows per CTA: groups of one, two
    and four CTAs share clusters, some with masked members."""
    ms = [1100, 1500, 600, 900, 330, 1090, 580] * 30
    masked = [3, 4, 20, 21, 55, 209]
    r = solve_batch(hn, torch_cuda, ms, masked=masked)
    for i in masked:
        assert np.array_equal(r[5][r[1][i]:r[1][i + 1]], r[4][r[1][i]:r[1][i + 1]])
    for i in [0, 1, 2, 5, 6, 57, 58, 60, 62, 207, 208]:
        check(i, *r, 1.0)
    assert np.array_equal(solve_batch(hn, torch_cuda, ms, masked=masked)[5], r[5])


@pytest.mark.parametrize("m", [1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64])
@pytest.mark.parametrize("scale", [1.0, 1e-140])
def test_largest_block(hn, torch_cuda, m, scale):
    """The diagonal blocks' kernel has as many rows as the step's largest block, 16 at a time."""
    for ms in ([m, 1, max(1, m - 1), m, 2], [64 + m, 64, 3]):
        r = solve_batch(hn, torch_cuda, ms, scale)
        for i in range(len(ms)):
            check(i, *r, scale)


@pytest.mark.parametrize("m", [1, 16, 17, 32, 33, 64, 65])
def test_instances_of_one_block(hn, torch_cuda, m):
    """A warp per instance up to 64 rows, beside the form for more (one of 65 rows
    in the batch); masked ones keep their right-hand sides."""
    ms, masked = [m, 1, max(1, m - 1), 2, m, max(1, m - 3)], [1, 4]
    for extra in ([], [65]):
        r = solve_batch(hn, torch_cuda, ms + extra, masked=masked)
        for i in range(len(ms)):
            if i in masked:
                assert np.array_equal(r[5][r[1][i]:r[1][i + 1]], r[4][r[1][i]:r[1][i + 1]])
            else:
                check(i, *r, 1.0)


def test_after_shutdown(hn, torch_cuda):
    """hn_shutdown gives memory and host words back, with a handle alive or
    without; the library goes on."""
    ms = [70, 3, 64]
    want = solve_batch(hn, torch_cuda, ms)[5]
    hn.check(hn.load().hn_shutdown())
    assert np.array_equal(solve_batch(hn, torch_cuda, ms)[5], want)
    lib, p64, h = hn.load(), C.POINTER(C.c_int64), C.c_void_p()
    A = hn.Csr(3, 3, [0, 1, 2, 4], [0, 1, 1, 2], [2.0, 1.0, 1.0, 1.0])
    P, ro = hn.Pattern(A), np.array([0, 3], np.int64)
    hn.check(lib.hn_batch_create(1, ro.ctypes.data_as(p64), ro.ctypes.data_as(p64), P.h, C.byref(h)))
    hn.check(lib.hn_shutdown())
    assert np.array_equal(solve_batch(hn, torch_cuda, ms)[5], want)
    hn.check(lib.hn_batch_destroy(h))
    hn.init(0)
