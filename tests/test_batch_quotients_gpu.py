"""GPU: the batched factorisation's quotients have the bits of IEEE division
(numpy's), by its own division where that holds and by CUDA's elsewhere:
random mantissas over the whole range, mantissas near one and near all ones,
the exponents at which the two ways meet, signed zeros, subnormals, infinities
and NaN, and reciprocals."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def doubles(rng, n, lo, hi):
    """Random signs and mantissas, exponents lo .. hi."""
    return np.ldexp(rng.uniform(1.0, 2.0, n) * rng.choice([-1.0, 1.0], n), rng.integers(lo, hi + 1, n))


def near_ones(rng, n):
    """1 + k ulps and 2 - k ulps for small k, exponents -3 .. 3."""
    k = rng.integers(0, 5, n)
    m = np.where(rng.random(n) < 0.5, 1.0 + k * 2.0**-52, 2.0 - k * 2.0**-52)
    return np.ldexp(m, rng.integers(-3, 4, n))


def pairs(kind, rng):
    n = 1 << 20
    if kind == "ordinary":
        return doubles(rng, n, -30, 30), np.abs(doubles(rng, n, -30, 30))
    if kind == "whole range":
        return doubles(rng, n, -1070, 1023), doubles(rng, n, -1070, 1023)
    if kind == "mantissas near one and two":
        return near_ones(rng, n) * rng.choice([-1.0, 1.0], n), near_ones(rng, n)
    if kind == "divisor of all ones":
        return doubles(rng, n, -5, 5), np.ldexp(np.full(n, 2.0 - 2.0**-52), rng.integers(-5, 6, n))
    if kind == "exact":  # a = q d without rounding: the residual is zero
        q, d = rng.integers(-(1 << 26), 1 << 26, n).astype(float), rng.integers(1, 1 << 26, n).astype(float)
        return q * d, d
    if kind == "reciprocal":
        return np.ones(n), doubles(rng, n, -410, 410)
    if kind == "ends of the range":  # 2^-400 and 2^401, from both sides
        e = np.array([-402, -401, -400, -399, 399, 400, 401, 402])
        return np.ldexp(doubles(rng, n, 0, 0), rng.choice(e, n)), np.ldexp(doubles(rng, n, 0, 0), rng.choice(e, n))
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.0**-1022, 2.0**-400, -2.0**-400,
                        np.nextafter(2.0**-400, 0), np.nextafter(2.0**401, 0), 2.0**401, 1.0, -1.0, 3.0, 1.7e308])
    a, d = np.meshgrid(special, special)
    return a.ravel(), d.ravel()


@pytest.mark.parametrize("kind", ["ordinary", "whole range", "mantissas near one and two", "divisor of all ones",
                                  "exact", "reciprocal", "ends of the range", "special values"])
def test_quotients_are_the_rounded_ones(hn, torch_cuda, kind):
    a, d = pairs(kind, np.random.default_rng(len(kind)))
    ad, dd = (torch_cuda.as_tensor(v, device="cuda") for v in (a, d))
    q = torch_cuda.full_like(ad, 7.0)
    hn.check(hn.load().hn_batch_quotients(a.size, ad.data_ptr(), dd.data_ptr(), q.data_ptr(), None))
    got = q.cpu().numpy()
    with np.errstate(all="ignore"):
        want = a / d
    same = (got.view(np.int64) == want.view(np.int64)) | (np.isnan(got) & np.isnan(want))
    assert same.all(), [(x.hex(), y.hex(), g.hex(), w.hex())
                        for x, y, g, w in zip(a[~same][:4], d[~same][:4], got[~same][:4], want[~same][:4])]
