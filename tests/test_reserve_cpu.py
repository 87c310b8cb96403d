"""What tdv_ctx_reserve asks an injected allocator for (no GPU: the addresses
are never used).  The byte volumes of the directions stored apart are asked for
only where a call of the reserved size may use them."""
import ctypes

import pytest

from thundervision_b200 import _lib as L


@pytest.fixture(scope="module")
def lib():
    L.build()
    return L.lib()


class Ctx:
    def __init__(self, lib, limit=1 << 60):
        self.lib, self.limit, self.asked, self.live, self.next = lib, limit, [], {}, 1 << 40
        self.h = ctypes.c_void_p()
        assert lib.tdv_ctx_create(0, ctypes.byref(self.h)) == L.TDV_OK
        self.fns = L.ALLOC_FN(self._alloc), L.FREE_FN(self._free)
        assert lib.tdv_ctx_set_allocator(self.h, *self.fns, None) == L.TDV_OK

    def _alloc(self, n, user):
        self.asked.append(n)
        if n > self.limit:
            return None
        p, self.next = self.next, self.next + (n + 4095) // 4096 * 4096
        self.live[p] = n
        return p

    def _free(self, p, user):
        del self.live[p]

    def reserve(self, W, H, D):
        self.asked.clear()
        assert self.lib.tdv_ctx_reserve(self.h, W, H, D) == L.TDV_OK
        return list(self.asked)

    def close(self):
        self.lib.tdv_ctx_destroy(self.h)


@pytest.fixture()
def make(lib):
    made = []

    def f(**kw):
        made.append(Ctx(lib, **kw))
        return made[-1]

    yield f
    for c in made:
        c.close()


def test_within_range(make):
    asked = make().reserve(1920, 1080, 256)
    # planes, two 16-bit volumes, the row scratch, eight byte volumes with the side words
    assert len(asked) == 5
    assert asked[1] == asked[2] == 1920 * 1080 * 256 * 2
    assert 8 * 1920 * 1080 * 256 <= asked[4] <= 8 * (1920 * 1080 * 260 + 256)


@pytest.mark.parametrize("W,H,D", [(4096, 4096, 256),   # one direction's volume reaches 4 GB: no call uses it
                                   (3840, 2160, 256)])  # eight take 17 GB
def test_no_volumes_no_call_can_use(make, W, H, D):
    asked = make().reserve(W, H, D)
    assert len(asked) == 4 and max(asked) == W * H * D * 2


def test_reserving_again_after_a_refusal(make):
    c = make(limit=1 << 30)
    assert len(c.reserve(1024, 768, 256)) >= 5 and len(c.live) == 4
    c.limit = 1 << 60
    c.reserve(1024, 768, 256)
    assert len(c.live) == 5
    # the refusal was no error of the call that met it
    assert c.lib.tdv_last_error_string(c.h) == b""


def test_smaller_reservation_keeps_what_is_there(make):
    c = make()
    c.reserve(800, 600, 128)
    live = dict(c.live)
    assert c.reserve(640, 480, 64) == [] and c.live == live
