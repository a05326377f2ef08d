"""GPU: the one-launch product of matrices of few tiles, against the two
launches of hn_spmv_noalloc, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def matrix(rows, n, rng):
    """CSR with the given row lengths, random columns (repeats allowed) and values."""
    rp = np.concatenate([[0], np.cumsum(rows)]).astype(np.int64)
    return rp, rng.integers(0, n, rp[-1]), rng.standard_normal(rp[-1])


def two_launches(hn, torch, m, n, rp, ci, val, x):
    dev = lambda a, t: torch.as_tensor(np.ascontiguousarray(a, t), device="cuda")  # noqa: E731
    y = torch.full((m,), np.nan, dtype=torch.float64, device="cuda")
    rpd, cid, vd = dev(rp, np.int32), dev(ci, np.int32), dev(val, np.float64)
    hn.check(hn.load().hn_spmv_noalloc(m, n, len(ci), rpd.data_ptr(), cid.data_ptr(), vd.data_ptr(), x.data_ptr(),
                                       y.data_ptr(), None))
    torch.cuda.synchronize()
    return y


def test_products_after_overlapping_ones(hn, torch_cuda):
    """Products of one handle on two streams may not overlap; where they did
    (no result of theirs is looked at), the next one alone is right again."""
    torch, rng = torch_cuda, np.random.default_rng(1)
    rows, n = np.array([1400, 600, 300] * 40), 10_000
    rp, ci, val = matrix(rows, n, rng)
    x = torch.as_tensor(rng.standard_normal(n), device="cuda")
    want = two_launches(hn, torch, rows.size, n, rp, ci, val, x)
    A = hn.Csr(rows.size, n, rp, ci, val, autotune=False)
    streams, ys = [torch.cuda.Stream() for _ in range(2)], [torch.empty_like(want) for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(400):
        for s, y in zip(streams, ys):
            A.spmv(x, y, stream=s.cuda_stream)
    torch.cuda.synchronize()
    y = torch.full_like(want, np.nan)
    for _ in range(3):
        A.spmv(x, y)
        assert torch.equal(y, want)


TILE = 1792  # row ends and entries of a merge-path tile


def tiles_of(n, kind):
    """Row lengths of exactly n tiles: rows of 15 entries (no head over 15), or of 3,583 (heads of 1,791)."""
    if kind == "short":
        return np.full(n * TILE // 16, 15)
    return np.full(n * TILE // 3584, 3583)


@pytest.mark.parametrize("n", [2, 4, 444, 446, 2046, 2048, 2050])
@pytest.mark.parametrize("kind", ["short", "long"])
def test_lines_between_one_launch_and_two(hn, torch_cuda, n, kind):
    """Up to 444 tiles (long heads) or 2,048 (short ones) one launch, the same bits on both sides of the lines."""
    torch, rng = torch_cuda, np.random.default_rng(n)
    rows, cols = tiles_of(n, kind), 5000
    rp, ci, val = matrix(rows, cols, rng)
    x = torch.as_tensor(rng.standard_normal(cols), device="cuda")
    A = hn.Csr(rows.size, cols, rp, ci, val, transpose=False, autotune=False)
    assert A.tiles()[1].size == n + 1
    want = two_launches(hn, torch, rows.size, cols, rp, ci, val, x)
    for _ in range(2):
        y, before = torch.full_like(want, np.nan), hn.stats()[0]
        A.spmv(x, y)
        assert hn.stats()[0] - before == (1 if n <= (2048 if kind == "short" else 444) else 2)
        assert torch.equal(y, want)


def rows_with_heads(h, extra, tiles):
    """Row lengths such that every tile after the first starts h entries into a row of h + extra."""
    rows, pos = [], 0
    for t in range(1, tiles):
        rows += [t * TILE - h - pos - 1, h + extra]
        pos = t * TILE + extra + 1
    return np.array(rows + [100])


def unique_columns(rows, n, rng):
    rp = np.concatenate([[0], np.cumsum(rows)]).astype(np.int64)
    ci = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in rows])
    return rp, ci, rng.standard_normal(ci.size)


@pytest.mark.parametrize("h", [1, 6, 7, 8, 255, 256, 257])
@pytest.mark.parametrize("extra", [0, 1, 44])
@pytest.mark.parametrize("special", [False, True])
def test_heads_up_to_the_limit(hn, torch_cuda, h, extra, special):
    """Carries recomputed up to 256 entries, by the ticket past them; as A x and
    as A^T x; with infinities and NaN among the values."""
    torch, rng = torch_cuda, np.random.default_rng(h + extra)
    rows, n = rows_with_heads(h, extra, 6), 3000
    rp, ci, val = unique_columns(rows, n, rng)
    m, xs = rows.size, rng.standard_normal(n)
    if special:
        xs[rng.integers(0, n, 3)] = [np.inf, -np.inf, np.nan]
        val[rng.integers(0, val.size, 2)] = [np.inf, -0.0]
    x = torch.as_tensor(xs, device="cuda")
    A = hn.Csr(m, n, rp, ci, val, autotune=False)
    _, row, nz = A.tiles()
    heads = [nz[t] - rp[row[t]] for t in range(1, len(row) - 1) if row[t] < m]
    assert len(heads) >= 5 and heads[:5] == [h] * 5
    want = two_launches(hn, torch, m, n, rp, ci, val, x)
    order = np.lexsort((np.repeat(np.arange(m), rows), ci))  # the transpose, whose A^T is this matrix
    rpT = np.concatenate([[0], np.cumsum(np.bincount(ci, minlength=n))])
    T = hn.Csr(n, m, rpT, np.repeat(np.arange(m), rows)[order], val[order], autotune=False)
    if special:  # exact zeros are left out of A^T
        keep = val != 0.0
        assert T.nnz_t == keep.sum()
    else:
        assert np.array_equal(T.tiles(trans=1)[1], row)
    for _ in range(2):
        for M, trans in ((A, 0), (T, 1)):
            y = torch.full((m,), np.nan, dtype=torch.float64, device="cuda")
            M.spmv(x, y, trans)
            if trans and special and T.nnz_t != val.size:
                continue
            assert torch.equal(torch.nan_to_num(y, 7.25), torch.nan_to_num(want, 7.25))
            assert torch.equal(y.isnan(), want.isnan())
