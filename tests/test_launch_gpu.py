"""GPU: kernels set up while their predecessors run. A chain of dependent
calls -- library kernels after one another, after other libraries' kernels,
after fills and copies, and across two streams -- gives the bits that it gives
with a synchronisation after every call, on the default stream, on a stream of
its own and replayed from a captured graph."""
import numpy as np
import pytest

import lpgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [30, 700, 40_000])
@pytest.mark.parametrize("how", ["default", "stream", "graph"])
def test_chain_of_launches(m, how):
    import hnb200 as hn
    import torch

    hn.init(0)
    n = 5 * m // 2
    lp = lpgen.lp_uniform(m, n, 6, 5)
    A = hn.Csr(m, n, lp["rp"], lp["ci"], lp["val"])
    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    x0 = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
    b = torch.randn(m, generator=g, dtype=torch.float64, device="cuda")
    other = torch.cuda.Stream()

    def chain(step):
        """step() after every call; buffers are new, so that nothing is left from a chain before."""
        x, y, r, t, u = x0.clone(), *(torch.full((k,), np.nan, dtype=torch.float64, device="cuda")
                                      for k in (m, m, n, n))
        out = torch.full((2,), np.nan, dtype=torch.float64, device="cuda")
        step()
        for _ in range(3):
            main = torch.cuda.current_stream()
            s = main.cuda_stream
            for call in (lambda: A.spmv(x, y, stream=s),                      # library after another's kernel
                         lambda: A.residual(x, b, r, stream=s),
                         lambda: hn.axpy(m, -0.5, y, r, stream=s),            # after two library kernels
                         lambda: t.zero_(),                                   # fill between
                         lambda: A.spmv(r, t, 1, 0.25, 1.0, stream=s),
                         lambda: u.copy_(t),                                  # copy between
                         lambda: hn.dot(n, t, u, out[:1].data_ptr(), stream=s),
                         lambda: u.mul_(1.0 / (1.0 + out[0]))):               # another's kernel after it
                call()
                step()
            other.wait_stream(main)
            with torch.cuda.stream(other):
                hn.dot(n, u, u, out[1:].data_ptr(), stream=other.cuda_stream)
                step()
            hn.axpy(n, 0.125, u, x, stream=s)
            step()
            main.wait_stream(other)
            hn.axpy(n, 0.125, t, u, stream=s)
            step()
        return x, y, r, t, u, out

    want = [v.clone() for v in chain(torch.cuda.synchronize)]
    if how == "graph":
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            chain(lambda: None)  # the workspace of a stream is made by its first call
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            got = chain(lambda: None)
        for _ in range(5):
            graph.replay()
            torch.cuda.synchronize()
            for a, w in zip(got, want):
                assert torch.equal(a, w)
        return
    stream = torch.cuda.Stream() if how == "stream" else torch.cuda.current_stream()
    for _ in range(5):
        with torch.cuda.stream(stream):
            got = chain(lambda: None)
        torch.cuda.synchronize()
        for a, w in zip(got, want):
            assert torch.isfinite(w).all() and torch.equal(a, w)
