"""GPU: threads with handles and streams of their own set models up, multiply,
assemble, select and solve at the same time; each gets what it gets alone."""
import ctypes as C
import threading

import numpy as np
import pytest

import lpgen

pytestmark = pytest.mark.gpu


def work(hn, torch, seed, reps):
    """Results of `reps` models of four sizes, on a stream of the thread's own."""
    lib, p64, results, stream = hn.load(), C.POINTER(C.c_int64), [], torch.cuda.Stream()
    dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
    with torch.cuda.stream(stream):
        s = stream.cuda_stream
        for r in range(reps):
            i = (seed + r) % 4
            m = [50, 300, 900, 2500][i]
            n, rng = 3 * m, np.random.default_rng(10 * seed + i)
            lp = lpgen.lp_uniform(m, n, 5, 10 * seed + i)
            A = hn.Csr(m, n, lp["rp"], lp["ci"], lp["val"], autotune=False)
            P = hn.Pattern(A)
            x, d = dev(rng.standard_normal(n)), dev(rng.uniform(0.5, 2, n))
            y, sol = (torch.empty(m, dtype=torch.float64, device="cuda") for _ in range(2))
            t, nval = (torch.empty(k, dtype=torch.float64, device="cuda") for k in (n, P.nnz))
            out = torch.empty(17, dtype=torch.int64, device="cuda")
            A.spmv(x, y, stream=s)
            A.spmv(y, t, 1, stream=s)
            hn.price_select(n, t, None, torch.arange(n, dtype=torch.int32, device="cuda"), None, out, k=16, stream=s)
            ro, co, h = np.array([0, m], np.int64), np.array([0, n], np.int64), C.c_void_p()
            hn.check(lib.hn_batch_create(1, ro.ctypes.data_as(p64), co.ctypes.data_as(p64), P.h, C.byref(h)))
            st = torch.zeros(1, dtype=torch.int32, device="cuda")
            hn.check(lib.hn_batch_factor(h, d.data_ptr(), 0.0, 1e-300, nval.data_ptr(), st.data_ptr(), s))
            hn.check(lib.hn_batch_solve(h, nval.data_ptr(), y.data_ptr(), sol.data_ptr(), st.data_ptr(), s))
            stream.synchronize()
            results.append([v.cpu().numpy() for v in (y, t, out, nval, sol)])
            hn.check(lib.hn_batch_destroy(h))
            P.close()
            A.close()
    return results


def test_threads_with_their_own_handles(hn, torch_cuda):
    want = [work(hn, torch_cuda, i, 4) for i in range(6)]
    got, errors = {}, []

    def run(i):
        try:
            got[i] = work(hn, torch_cuda, i, 12)
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    ts = [threading.Thread(target=run, args=(i,)) for i in range(6)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors, errors[:2]
    for i, results in got.items():
        for r, values in enumerate(results):
            assert all(np.array_equal(a, b) for a, b in zip(values, want[i][r % 4]))
