"""GPU: hn_malloc / hn_free and the handles' memory behave as cudaMalloc and
cudaFree do, whatever the cache of freed blocks holds."""
import ctypes as C

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
