"""GPU: infinities, NaN, signed zeros and the type's extremes in the SpMM and in
the pricing selection, against the same operations in numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same_bits(a, b):
    return np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(
        np.where(np.isnan(a), 0.0, a).view(np.int64), np.where(np.isnan(b), 0.0, b).view(np.int64))


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65])
def test_spmm(hn, torch_cuda, k):
    """C[i, :] = sum of a_ij B[j, :] in CSR order, each product and sum rounded."""
    rng = np.random.default_rng(k)
    rows, n = np.array([0, 1, 2, 3, 4, 5, 7, 8, 9, 33, 130, 0, 1, 12]), 200
    rp = np.concatenate([[0], np.cumsum(rows)])
    ci, val = rng.integers(0, n, rp[-1]), rng.standard_normal(rp[-1])
    B = rng.standard_normal((n, k))
    special = [np.inf, -np.inf, np.nan, -0.0, 0.0, 1.7e308, -1.7e308, 5e-324]
    B.ravel()[rng.integers(0, n * k, 24)] = special * 3
    val[rng.integers(0, val.size, 8)] = [np.inf, -0.0, 1e308, -1e308, 5e-324, 1e-308, np.nan, -np.inf]
    want = np.zeros((rows.size, k))
    with np.errstate(all="ignore"):
        for i in range(rows.size):
            for p in range(rp[i], rp[i + 1]):
                want[i] += val[p] * B[ci[p]]
    A = hn.Csr(rows.size, n, rp, ci, val, transpose=False)
    C = torch_cuda.full((rows.size, k), 3.0, dtype=torch_cuda.float64, device="cuda")
    A.spmm(torch_cuda.as_tensor(B, device="cuda"), k, C)
    assert same_bits(C.cpu().numpy(), want)


@pytest.mark.parametrize("n", [40, 4096, 60_000, 700_001])
@pytest.mark.parametrize("maximize", [False, True])
def test_selection(hn, torch_cuda, n, maximize):
    """The ranking by |rc| / sqrt(w), weights that are not positive and finite
    counting as 1, ties by the lower index; a score of zero counts and never places."""
    rng, tol = np.random.default_rng(n), 0.0
    rc, w = rng.standard_normal(n), rng.uniform(0.25, 4.0, n)
    at = lambda c: rng.integers(0, n, c)  # noqa: E731
    rc[at(12)] = [np.inf, -np.inf, np.nan, -0.0, 0.0, -5e-324, 1.7e308, -1.7e308, -np.inf, np.inf, -1e-300, 1e-300]
    w[at(10)] = [np.inf, -1.0, 0.0, np.nan, 5e-324, 1.7e308, -np.inf, -0.0, 1e-300, 1e300]
    i = at(6)
    rc[i], w[i] = (5e-324 if maximize else -5e-324), 1.7e308  # a score that rounds to zero
    nonbasis = np.where(rng.random(n) < 0.1, -1, np.arange(n)).astype(np.int32)
    with np.errstate(all="ignore"):
        r = -rc if maximize else rc
        eligible = (nonbasis >= 0) & (r < -tol)
        score = np.where(eligible, np.abs(r) / np.sqrt(np.where((w > 0) & np.isfinite(w), w, 1.0)), 0.0)
    order = np.lexsort((np.arange(n), -score))
    order = order[score[order] > 0.0]
    dev = lambda a: torch_cuda.as_tensor(a, device="cuda")  # noqa: E731
    for k in (1, 3, 16, 64):
        out = torch_cuda.full((k + 1,), 77, dtype=torch_cuda.int64, device="cuda")
        hn.price_select(n, dev(rc), dev(w), dev(nonbasis), None, out, maximize=maximize, tol=tol, k=k)
        want = np.full(k, -1)
        want[:min(k, order.size)] = order[:k]
        assert out.cpu().tolist() == [eligible.sum(), *want]
    out = torch_cuda.full((2,), 77, dtype=torch_cuda.int64, device="cuda")
    hn.price_select(n, dev(rc), dev(w), dev(nonbasis), None, out, maximize=maximize, tol=tol, rule=hn.PRICE_BLAND)
    assert out.cpu().tolist() == [eligible.sum(), np.flatnonzero(eligible)[0] if eligible.any() else -1]
