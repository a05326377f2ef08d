"""GPU: the backend's resident matrices are found by their contents, wherever
the arrays lie (the C interface copies them, a thread's copies come from its
own arena), uploads are counted in kernel launches."""
import threading

import numpy as np
import pytest

import lpgen
import oracle as O

pytestmark = pytest.mark.gpu


def in_thread(f):
    out = []
    t = threading.Thread(target=lambda: out.append(f()))
    t.start()
    t.join()
    return out[0]


def launches(be, f):
    before = be.kernel_executions()
    y = f()
    return be.kernel_executions() - before, y


def test_found_at_another_address(hn):
    be, lp = hn.Backend(), lpgen.lp_uniform(300, 900, 4, 3)
    rp, ci, val, x = lp["rp"], lp["ci"], lp["val"], np.ones(900)
    call = lambda v=val: launches(be, lambda: be.spmv(rp, ci, v, x))  # noqa: E731
    first, y = call()
    resident, y2 = call()
    assert resident < first and np.array_equal(y, y2)
    for _ in range(3):
        n, yt = in_thread(call)
        assert n == resident and np.array_equal(y, yt)
        assert call()[0] == resident
    n, y3 = in_thread(lambda: call(2.0 * val))  # other contents are another matrix
    assert n == first and np.array_equal(y3, 2.0 * y)
    assert in_thread(lambda: call(2.0 * val))[0] == resident
    be.close()


def test_columns_without_entries(hn):
    """The same entries with more or fewer empty columns behind them, whichever came first."""
    be, lp = hn.Backend(), lpgen.lp_uniform(40, 60, 4, 3)
    rp, ci, val = lp["rp"], lp["ci"], lp["val"]
    used = int(max(ci)) + 1
    for n in (used + 40, used, used + 7, used + 40):
        x = np.arange(1.0, n + 1)
        np.testing.assert_allclose(be.spmv(rp, ci, val, x), O.multiply(rp, ci, val, x), rtol=1e-12)
        t = be.spmv_t(rp, ci, val, np.ones(40), n)
        assert t.shape == (n,)
        np.testing.assert_allclose(t, O.tmultiply(rp, ci, val, np.ones(40), n), rtol=1e-12, atol=1e-300)
    be.close()


def test_many_matrices(hn):
    """More matrices than are kept: each product is its own, and those used last are resident."""
    be, lp = hn.Backend(), lpgen.lp_uniform(50, 100, 3, 3)
    rp, ci, x = lp["rp"], lp["ci"], np.ones(100)
    y = be.spmv(rp, ci, lp["val"], x)
    for i in range(40):
        f = lambda: be.spmv(rp, ci, 2.0**(i % 20) * lp["val"], x)  # noqa: E731, B023
        assert np.array_equal(in_thread(f) if i % 2 else f(), 2.0**(i % 20) * y)
    be.close()
