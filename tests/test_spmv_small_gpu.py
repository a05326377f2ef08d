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
