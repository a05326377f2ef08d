"""GPU: revised-simplex pricing on the device against the oracle's
restatement of SimplexSolver's pricing (pinned to the reference in
test_price.py): reduced costs and Devex weights bit-identical, the entering
choice and the ranked shortlist identical (ties by lower index), dense columns
equal to extract_column."""
import numpy as np
import pytest

import lpgen
import oracle as O
from test_price import pricing_state

pytestmark = pytest.mark.gpu


def dev(torch, a, dtype=None):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda", dtype=dtype)


@pytest.mark.parametrize("shape", [(120, 300, 7), (2000, 5000, 21)])
def test_reduced_costs_bit_exact(hn, torch_cuda, shape):
    torch = torch_cuda
    m, n, seed = shape
    lp, y, cost, *_ = pricing_state(m, n, seed)
    A = hn.Csr(lp["m"], lp["n"], lp["rp"], lp["ci"], lp["val"])
    rc = torch.empty(n, dtype=torch.float64, device="cuda")
    hn.price_reduced_costs(A, dev(torch, y), dev(torch, cost), rc)
    torch.cuda.synchronize()
    want = O.price_reduced_costs(m, n, lp["rp"], lp["ci"], lp["val"], y, cost)
    assert np.array_equal(rc.cpu().numpy(), want)


@pytest.mark.parametrize("zero_u", [False, True])
def test_devex_update_bit_exact(hn, torch_cuda, zero_u):
    torch = torch_cuda
    lp, y, cost, nonbasis, artificial, w = pricing_state(400, 1000, 13)
    w = np.abs(np.nan_to_num(w, nan=1.0, posinf=1.0))
    u = np.zeros(lp["m"]) if zero_u else np.random.default_rng(4).standard_normal(lp["m"])
    u[::5] = 0.0
    A = hn.Csr(lp["m"], lp["n"], lp["rp"], lp["ci"], lp["val"])
    wd = dev(torch, w)
    alpha = torch.empty(lp["n"], dtype=torch.float64, device="cuda")
    hn.price_devex_update(A, dev(torch, u), dev(torch, nonbasis), wd, alpha)
    torch.cuda.synchronize()
    want_w, want_alpha = O.price_devex_update(lp["m"], lp["n"], lp["rp"], lp["ci"], lp["val"], u, nonbasis, w)
    assert np.array_equal(alpha.cpu().numpy(), want_alpha)
    assert np.array_equal(wd.cpu().numpy(), want_w)


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("phase1,maximize", [(False, False), (True, False), (False, True)])
def test_select_matches_ranked_candidates(hn, torch_cuda, ties, phase1, maximize):
    torch = torch_cuda
    lp, y, cost, nonbasis, artificial, w = pricing_state(300, 800, 5, ties=ties)
    rc = O.price_reduced_costs(lp["m"], lp["n"], lp["rp"], lp["ci"], lp["val"], y, cost)
    if ties:
        rc = np.round(rc * 4) / 4
    n = lp["n"]
    args = (dev(torch, rc), dev(torch, w), dev(torch, nonbasis), dev(torch, artificial))
    k = 16
    out = torch.empty(k + 1, dtype=torch.int64, device="cuda")
    hn.price_select(n, *args, out, phase1=phase1, maximize=maximize, rule=hn.PRICE_RANKED, k=k)
    got = out.cpu().numpy()
    cnt, order = O.price_ranked(rc, w, nonbasis, artificial, phase1, maximize, cap=k)
    assert got[0] == cnt and cnt > k
    assert np.array_equal(got[1:], order)
    hn.price_select(n, *args, out, phase1=phase1, maximize=maximize, rule=hn.PRICE_BLAND)
    got = out.cpu().numpy()
    assert got[0] == cnt and got[1] == O.price_bland(rc, nonbasis, artificial, phase1, maximize)


def test_select_edge_cases(hn, torch_cuda):
    torch = torch_cuda
    n = 1000
    rng = np.random.default_rng(2)
    rc = np.abs(rng.standard_normal(n))  # nothing improving
    nb = np.arange(n, dtype=np.int32)
    out = torch.empty(5, dtype=torch.int64, device="cuda")
    hn.price_select(n, dev(torch, rc), None, dev(torch, nb), None, out, rule=hn.PRICE_RANKED, k=4)
    assert out.cpu().tolist() == [0, -1, -1, -1, -1]
    hn.price_select(n, dev(torch, rc), None, dev(torch, nb), None, out, rule=hn.PRICE_BLAND)
    assert out.cpu().tolist()[:2] == [0, -1]
    rc[[3, 700]] = -1.0  # two improving columns with equal score: index order
    hn.price_select(n, dev(torch, rc), None, dev(torch, nb), None, out, rule=hn.PRICE_RANKED, k=4)
    assert out.cpu().tolist() == [2, 3, 700, -1, -1]
    with pytest.raises(hn.HnError):
        hn.price_select(n, dev(torch, rc), None, dev(torch, nb), None, out, rule=hn.PRICE_RANKED, k=0)
    # empty problem
    hn.price_select(0, None, None, None, None, out, rule=hn.PRICE_RANKED, k=1)
    assert out.cpu().tolist()[:2] == [0, -1]


def test_columns_match_extract_column(hn, torch_cuda):
    torch = torch_cuda
    lp = lpgen.lp_uniform(500, 1250, 6, 8)
    A = hn.Csr(lp["m"], lp["n"], lp["rp"], lp["ci"], lp["val"])
    cols = np.array([0, 5, 1249, 600, 5], dtype=np.int64)
    out = torch.full((cols.size, lp["m"]), np.nan, dtype=torch.float64, device="cuda")
    hn.price_columns(A, dev(torch, cols), out)
    got = out.cpu().numpy()
    for r, j in enumerate(cols):
        assert np.array_equal(got[r], O.extract_column(lp["m"], lp["rp"], lp["ci"], lp["val"], int(j)))
    bad = dev(torch, np.array([1, 1250], dtype=np.int64))
    with pytest.raises(hn.HnError):
        hn.price_columns(A, bad, out[:2])


@pytest.mark.parametrize("n,k,improving", [(1, 1, 1), (511, 64, 300), (4096, 16, 4000), (4097, 64, 3000),
                                           (8192 + 3, 7, 5), (700_001, 64, 200_000), (700_001, 3, 1)])
def test_select_chunk_edges(hn, torch_cuda, n, k, improving):
    """Sizes around a block's chunk (4,096 columns) and past 148 blocks, few
    and many improving columns, repeated scores: order (score descending,
    index ascending), exact."""
    rng = np.random.default_rng(n + k)
    rc = np.abs(rng.standard_normal(n))
    rc[rng.permutation(n)[:improving]] = -np.round(rng.uniform(1.0, 3.0, improving), 3)
    w = rng.choice([1.0, 4.0, 0.25], n)
    nb = np.arange(n, dtype=np.int32)
    out = torch_cuda.empty(k + 1, dtype=torch_cuda.int64, device="cuda")
    args = (dev(torch_cuda, rc), dev(torch_cuda, w), dev(torch_cuda, nb), None, out)
    hn.price_select(n, *args, rule=hn.PRICE_RANKED, k=k)
    got = out.cpu().numpy()
    score = np.where(rc < -1e-9, np.abs(rc) / np.sqrt(w), 0.0)
    want = np.lexsort((np.arange(n), -score))[:min(k, improving)]
    assert got[0] == improving
    assert np.array_equal(got[1:1 + want.size], want) and np.all(got[1 + want.size:] == -1)
    hn.price_select(n, *args, rule=hn.PRICE_BLAND)
    assert out.cpu().tolist()[:2] == [improving, int(np.flatnonzero(rc < -1e-9)[0])]


@pytest.mark.parametrize("m", [1, 8191, 8192, 8193, 20_000])
def test_columns_row_slices(hn, torch_cuda, m):
    """Rows around the gather's slice of 8,192."""
    lp = lpgen.lp_uniform(m, 40, min(m, 9), 3)
    A = hn.Csr(m, 40, lp["rp"], lp["ci"], lp["val"])
    cols = np.array([39, 0, 17], dtype=np.int64)
    out = torch_cuda.full((3, m), np.nan, dtype=torch_cuda.float64, device="cuda")
    hn.price_columns(A, dev(torch_cuda, cols), out)
    for r, j in enumerate(cols):
        assert np.array_equal(out[r].cpu().numpy(), O.extract_column(m, lp["rp"], lp["ci"], lp["val"], int(j)))
