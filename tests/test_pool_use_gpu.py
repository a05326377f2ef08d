"""GPU: hn_malloc / hn_free and the handles' memory behave as cudaMalloc and
cudaFree do, whatever the cache of freed blocks holds."""
import ctypes as C
import threading

import pytest

pytestmark = pytest.mark.gpu

OUT_OF_MEMORY = 3


def alloc(hn, n):
    p = C.c_void_p()
    hn.check(hn.load().hn_malloc(C.byref(p), n))
    return p


@pytest.mark.parametrize("size", [2**64 - 1, 2**64 - 511, 2**64 - 512, 2**63, 2**62])
def test_sizes_past_the_address_space(hn, size):
    """Rounding such a size up does not make it a small one."""
    hn.check(hn.load().hn_free(alloc(hn, 1)))  # a small block is there to be had
    p = C.c_void_p()
    assert hn.load().hn_malloc(C.byref(p), size) == OUT_OF_MEMORY and not p.value


def capture(torch, mode, body):
    """x += 1, body(), x += 1 in a captured graph; x after one replay."""
    x, side = torch.zeros(8, device="cuda"), torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side, capture_error_mode=mode):
        x.add_(1)
        body()
        x.add_(1)
    graph.replay()
    torch.cuda.synchronize()
    return x[0].item()


@pytest.mark.parametrize("mode,other_thread", [("relaxed", False), ("relaxed", True), ("thread_local", True)])
@pytest.mark.parametrize("what", ["block", "set-up"])
def test_free_beside_a_capture(hn, torch_cuda, mode, other_thread, what):
    """Where cudaFree may run beside a capture, so may hn_free and a set-up with
    its temporaries: they succeed, the graph is whole and no error is left over."""
    if what == "block":
        p = alloc(hn, 1 << 20)
        call = lambda: hn.load().hn_free(p)  # noqa: E731
    else:
        kept = []  # a handle's end synchronises the device

        def call():
            kept.append(hn.Csr(2, 2, [0, 1, 2], [0, 1], [1.0, 2.0]))
            return 0

    got = []

    def body():
        if other_thread:
            t = threading.Thread(target=lambda: got.append(call()))
            t.start()
            t.join()
        else:
            got.append(call())

    assert capture(torch_cuda, mode, body) == 2.0
    assert got == [0]
    y = torch_cuda.ones(4, dtype=torch_cuda.float64, device="cuda")
    hn.axpy(4, 1.0, y, y.clone())  # the next launch has nothing else to report


def test_free_waits_for_every_stream(hn, torch_cuda):
    """A block comes back only after the work that uses it, on any stream."""
    n, s = 1 << 20, torch_cuda.cuda.Stream()
    p = alloc(hn, n)
    with torch_cuda.cuda.stream(s):
        torch_cuda.cuda._sleep(20_000_000)  # about 10 ms
    hn.check(hn.load().hn_memset(p, 1, n, s.cuda_stream))
    hn.check(hn.load().hn_free(p))
    assert s.query()
