"""GPU: the cache of freed device blocks behind hn_malloc / hn_free and the handles."""
import ctypes as C
import threading

import pytest

pytestmark = pytest.mark.gpu


def alloc(hn, n):
    p = C.c_void_p()
    hn.check(hn.load().hn_malloc(C.byref(p), n))
    return p


def test_double_free_is_an_error(hn):
    p = alloc(hn, 1000)
    hn.check(hn.load().hn_free(p))
    with pytest.raises(hn.HnError):
        hn.check(hn.load().hn_free(p))
    hn.check(hn.load().hn_free(None))


@pytest.mark.parametrize("size", [1, 511, 512, 513, 1 << 20, (256 << 20) + 1])
def test_blocks_do_not_overlap(hn, torch_cuda, size):
    """Live blocks are distinct, reused ones too, at the rounding and the size limit."""
    lib = hn.load()
    for _ in range(3):
        ps = sorted(alloc(hn, s).value for s in (size, size, max(1, size - 1), size + 1))
        assert all(b - a >= size - 1 for a, b in zip(ps, ps[1:])) and len(set(ps)) == 4
        for p in ps:
            hn.check(lib.hn_free(C.c_void_p(p)))


def test_threads(hn):
    """Each thread's bytes stay its own while others allocate and free."""
    lib, errors = hn.load(), []

    def work(t):
        try:
            for i in range(60):
                n = 1000 + 64 * ((t * 7 + i) % 50)
                p, back = alloc(hn, n), (C.c_ubyte * n)()
                hn.check(lib.hn_memset(p, t + 1, n, None))
                hn.check(lib.hn_memcpy_d2h(back, p, n, None))
                assert set(bytes(back)) == {t + 1}
                hn.check(lib.hn_free(p))
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    ts = [threading.Thread(target=work, args=(t,)) for t in range(8)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors, errors


def test_old_blocks_make_room(hn):
    """Freed blocks past the cache's size push the oldest out, and the newest stay."""
    lib = hn.load()
    big = [alloc(hn, (200 << 20) + 4096 * i) for i in range(7)]
    for p in big:
        hn.check(lib.hn_free(p))
    for n in (777 << 10, 255 << 20):
        p = alloc(hn, n)
        hn.check(lib.hn_free(p))
        q = alloc(hn, n)
        assert q.value == p.value
        hn.check(lib.hn_free(q))
    for p in big:
        with pytest.raises(hn.HnError):  # idle or gone
            hn.check(lib.hn_free(p))
