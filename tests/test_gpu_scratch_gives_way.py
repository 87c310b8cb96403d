"""Scratch that only speeds calls up gives way: a context whose allocator has a
fixed budget runs every call whose necessary scratch fits it, whatever calls
came before."""
import numpy as np
import pytest
import torch

from thundervision_b200 import api

pytestmark = pytest.mark.gpu

W, H, D = 300, 200, 64
CELLS = W * H * D


class Budget:
    def __init__(self, total):
        self.total, self.live, self.sizes = total, {}, {}
        self.ctx = api.Context(0)
        self.ctx.set_allocator(self._alloc, self._free)

    def _alloc(self, n, user):
        if sum(self.sizes.values()) + n > self.total:
            return None
        t = torch.empty(n, dtype=torch.uint8, device="cuda")
        self.live[t.data_ptr()], self.sizes[t.data_ptr()] = t, n
        return t.data_ptr()

    def _free(self, p, user):
        self.live.pop(p)
        self.sizes.pop(p)


def _pair(w, h, seed=2):
    rng = np.random.default_rng(seed)
    return [torch.from_numpy(rng.integers(0, 256, size=(h, w)).astype(np.uint8)).cuda() for _ in range(2)]


def _equal(a, b):
    return torch.equal(a["disp"].to(torch.int32), b["disp"].to(torch.int32))


def test_sgm_volume_before_the_passes_volumes(ctx):
    """Room for the aggregation volume and the schedule, and less than two volumes more."""
    cost = ctx.cost(*_pair(W, H), D)
    b = Budget(int(2.5 * CELLS * 4))
    for kw in ({}, dict(table="ref", semantics="ref_gpu")):
        assert _equal(b.ctx.sgm(cost, 10, 120, **kw), ctx.sgm(cost, 10, 120, **kw))
    b.ctx.close()


def test_fused_volumes_give_way(ctx):
    small, large = _pair(W, H // 2), _pair(W, H, 3)
    # the small pair's two 16-bit and eight byte volumes, or the large pair's two
    b = Budget(2 * CELLS + 4 * CELLS + (3 << 20))
    for _ in range(2):
        assert _equal(b.ctx.stereo_sgm(*small, D, 10, 120, lr=1), ctx.stereo_sgm(*small, D, 10, 120, lr=1))
    assert max(b.sizes.values()) >= 4 * CELLS  # holds byte volumes
    assert _equal(b.ctx.stereo_sgm(*large, D, 10, 120, lr=1), ctx.stereo_sgm(*large, D, 10, 120, lr=1))
    b.ctx.close()


def test_batch_takes_their_place(ctx):
    pair = _pair(W, H)
    # the call's two 16-bit and eight byte volumes, or those two beside the batch's
    b = Budget(4 * CELLS + 8 * CELLS + (6 << 20))
    assert _equal(b.ctx.stereo_sgm(*pair, D, 10, 120), ctx.stereo_sgm(*pair, D, 10, 120))
    assert max(b.sizes.values()) >= 8 * CELLS
    batch = api.Batch(b.ctx, [(*pair, D, None)], 10, 300)
    assert _equal(batch.run()[0], ctx.stereo_sgm(*pair, D, 10, 300))
    batch.status()
    batch.close()
    b.ctx.close()
