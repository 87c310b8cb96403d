"""tdv_batch_autotune on batches that store the directions apart: only the
queue order is a candidate, so every other field stays as it was set."""
import numpy as np
import pytest
import torch

from thundervision_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [0, 1])
def test_only_the_order(ctx, order):
    rng = np.random.default_rng(1)
    pairs = []
    for W, H, D in [(200, 90, 64), (96, 64, 16), (300, 40, 128)]:
        l, r = [torch.from_numpy(rng.integers(0, 256, size=(H, W)).astype(np.uint8)).cuda() for _ in range(2)]
        pairs.append((l, r, D, 1))
    b = api.Batch(ctx, pairs, 10, 120)
    set_to = dict(lines_per_cta=5, rows_per_cta=3, split_disparity=1, order=order, ctas_per_sm=2)
    b.set_tiles(**set_to)
    tiles, ms = b.autotune(reps=1)
    assert ms > 0 and np.isfinite(ms)
    assert {k: v for k, v in tiles.items() if k != "order"} == {k: v for k, v in set_to.items() if k != "order"}
    assert b.tiles == tiles
    out = b.run()
    b.status()
    for (l, r, D, lr), o in zip(pairs, out):
        want = ctx.stereo_sgm(l, r, D, 10, 120, lr=lr)["disp"]
        assert torch.equal(o["disp"].to(torch.int32), want.to(torch.int32))
    b.close()
