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
