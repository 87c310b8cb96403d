"""Calls within a reserved size allocate and release nothing, also where the
reservation's byte volumes were refused, and give the same maps."""
import numpy as np
import pytest
import torch

from thundervision_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("refused", [True, False])
def test_no_allocation_within_a_reservation(refused):
    W, H, D = 300, 200, 64
    live, calls = {}, []

    def alloc(n, user):
        calls.append(("alloc", n))
        if refused and n > 2 * W * H * D + (1 << 20):
            return None
        t = torch.empty(n, dtype=torch.uint8, device="cuda")
        live[t.data_ptr()] = t
        return t.data_ptr()

    def release(p, user):
        calls.append(("release", p))
        live.pop(p)

    c, plain = api.Context(0), api.Context(0)
    try:
        c.set_allocator(alloc, release)
        c.reserve(W, H, D)
        rng = np.random.default_rng(2)
        pairs = []
        for w, h, d in [(60, 40, 16), (100, 80, 33), (W, 80, 64), (W, H, 48), (W, H, D)]:
            l, r = [torch.from_numpy(rng.integers(0, 256, size=(h, w)).astype(np.uint8)).cuda() for _ in range(2)]
            pairs.append((l, r, d))
        c.stereo_sgm(*pairs[0], 10, 120)  # the error word
        calls.clear()
        names = []
        for l, r, d in pairs:
            out = []
            names += [n for n, _ in c.kernel_times(lambda: out.append(c.stereo_sgm(l, r, d, 10, 120, lr=1)))]
            want = plain.stereo_sgm(l, r, d, 10, 120, lr=1)["disp"]
            assert torch.equal(out[0]["disp"].to(torch.int32), want.to(torch.int32))
        assert calls == []
        assert ("fused_sum_wta" in names) == (not refused)
    finally:
        torch.cuda.synchronize()
        c.close()
        plain.close()
