"""The general aggregation's padded runs: ranges that are no multiple of 8 with
the passes in groups of two, and scratch that does not start on 32 bytes (the
passes then run in sequence), bit-exact against the oracle."""
import numpy as np
import pytest
import torch

from thundervision_b200 import api

pytestmark = pytest.mark.gpu


def _context(limit, offset):
    live = {}

    def alloc(n, user):
        if n > limit:
            return None
        t = torch.empty(n + offset, dtype=torch.uint8, device="cuda")
        live[t.data_ptr() + offset] = t
        return t.data_ptr() + offset

    c = api.Context(0)
    c.set_allocator(alloc, lambda p, user: live.pop(p, None))
    return c


@pytest.mark.parametrize("groups,offset", [(True, 0), (False, 0), (False, 16)])
@pytest.mark.parametrize("sem,table", [("standard", "full"), ("ref_cpu", "ref"), ("ref_gpu", "ref")])
@pytest.mark.parametrize("D", [5, 37, 63, 100])
def test_padded_runs(orc, groups, offset, sem, table, D):
    W, H = 61, 43
    vol = (W * H * ((D + 7) // 8 * 8) * 4 + 255) // 256 * 256
    ctx = _context(2 * vol if groups else 1 << 40, offset)
    try:
        rng = np.random.default_rng(D)
        C = rng.uniform(0, 3, size=(H, W, D)).astype(np.float32)
        for x in range(min(W, D)):
            C[:, x, x + 1:] = np.inf
        guide = rng.integers(0, 5, size=(H, W)).astype(np.float32) / 4
        d, _, S = orc.sgm(C, guide, 0.3, 1.7, p2_mode=1, paths=8, table={"full": 0, "ref": 1}[table],
                          semantics={"standard": 0, "ref_cpu": 1, "ref_gpu": 2}[sem])
        agg = torch.empty((H, W, D), device="cuda")
        out = ctx.sgm(torch.from_numpy(C).cuda(), 0.3, 1.7, guide=torch.from_numpy(guide).cuda(), p2_mode="adjust",
                      table=table, semantics=sem, aggreg=agg)
        np.testing.assert_array_equal(agg.cpu().numpy(), S)
        np.testing.assert_array_equal(out["disp"].cpu().numpy(), d)
    finally:
        torch.cuda.synchronize()
        ctx.close()
