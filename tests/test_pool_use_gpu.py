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


@pytest.fixture
def cudart(torch_cuda):
    """The CUDA runtime that torch loaded: another user of the same device."""
    rt = C.CDLL("libcudart.so.12")
    rt.cudaMalloc.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]
    rt.cudaFree.argtypes = [C.c_void_p]
    yield rt
    rt.cudaGetLastError()


def test_block_freed_past_the_library(hn, cudart):
    """cudaFree on a block of hn_malloc: the library does not take the address
    for its block any more, freed or not, nor hand it out."""
    lib, n = hn.load(), 3 << 20
    p = alloc(hn, n)
    assert cudart.cudaFree(p) == 0
    assert lib.hn_free(p) != 0  # nothing there to free
    idle = alloc(hn, n)
    hn.check(lib.hn_free(idle))
    assert cudart.cudaFree(idle) == 0
    q, back = alloc(hn, n), (C.c_ubyte * n)()
    hn.check(lib.hn_memset(q, 5, n, None))
    hn.check(lib.hn_memcpy_d2h(back, q, n, None))
    assert set(bytes(back)) == {5}
    hn.check(lib.hn_free(q))
    assert lib.hn_free(q) != 0


@pytest.mark.parametrize("size", [3 << 20, 2 << 20, 4 << 20])
@pytest.mark.parametrize("state", ["live", "idle"])
def test_address_given_to_another(hn, cudart, size, state):
    """A block of 3 MB was freed past the library and the driver gave its
    address to another allocation: hn_free frees that one, as cudaFree does."""
    lib, n, others = hn.load(), 3 << 20, []
    p = alloc(hn, n)
    if state == "idle":
        hn.check(lib.hn_free(p))
    assert cudart.cudaFree(p) == 0
    for _ in range(8):
        q = C.c_void_p()
        assert cudart.cudaMalloc(C.byref(q), size) == 0
        others.append(q)
    hn.check(lib.hn_memset(others[0], 1, size, None))
    if state == "idle":  # not handed out while another has it
        r = alloc(hn, n)
        assert all(abs(r.value - q.value) >= min(n, size) for q in others)
        hn.check(lib.hn_free(r))
    for q in others:
        hn.check(lib.hn_free(q))
        assert cudart.cudaFree(q) != 0  # gone, not kept


def test_a_threads_first_call(hn):
    """A thread whose first call this is finds the freed blocks, and double frees."""
    lib, n, got = hn.load(), 5 << 20, []
    p = alloc(hn, n)
    hn.check(lib.hn_free(p))
    for call in (lambda: got.append(alloc(hn, n).value), lambda: got.append(lib.hn_free(p)),
                 lambda: got.append(lib.hn_free(p) != 0)):
        t = threading.Thread(target=call)
        t.start()
        t.join()
    assert got == [p.value, 0, True]


def test_freed_memory_is_free(hn, torch_cuda):
    """free_mem after a free is what it was before the allocation, and after
    hn_trim the device has the memory for everybody."""
    lib, n = hn.load(), 200 << 20
    device_free = lambda: torch_cuda.cuda.mem_get_info()[0]  # noqa: E731
    hn.check(lib.hn_trim())
    before = hn.device_info().free_mem
    assert before == device_free()
    p = alloc(hn, n)
    assert hn.device_info().free_mem <= before - n
    hn.check(lib.hn_free(p))
    assert hn.device_info().free_mem == before
    hn.check(lib.hn_trim())
    assert hn.device_info().free_mem == before == device_free()
    q = alloc(hn, n)  # and goes on
    hn.check(lib.hn_free(q))
