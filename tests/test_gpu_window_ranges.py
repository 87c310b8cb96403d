"""Window costs at the edges of their tile rules, bit-exact against the oracle:
narrow ranges (one row per item, runs of 8 pixels), ranges so wide that a tile
has 4 or 2 rows, and the fused Gaussian over more columns than it filters at a
time."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

KIND_ID = {"bt": 0, "ssd": 1, "ncc": 2}


def _pair(W, H, seed):
    rng = np.random.default_rng(seed)
    L, R = [rng.random((H, W), dtype=np.float32) for _ in range(2)]
    L[:, : W // 5] = 0.5
    R[: H // 3, : W // 4] = 0.0
    return L, R


def _check(ctx, orc, kind, radius, W, H, D):
    L, R = _pair(W, H, W + D + radius)
    Lt, Rt = torch.from_numpy(L).cuda(), torch.from_numpy(R).cuda()
    C = ctx.cost(Lt, Rt, D, kind=kind, radius=radius)
    assert np.array_equal(C.cpu().numpy(), orc.cost_pair(L, R, D, KIND_ID[kind], radius, orc.LAYOUT_HWD),
                          equal_nan=True)
    F, left = ctx.cost_filtered(Lt, Rt, D, kind=kind, radius=radius)
    fl, fr = ctx.prefilter(Lt), ctx.prefilter(Rt)
    assert torch.equal(left, fl)
    want = ctx.cost(fl, fr, D, kind=kind, radius=radius)
    assert np.array_equal(F.cpu().numpy(), want.cpu().numpy(), equal_nan=True)


@pytest.mark.parametrize("radius", [1, 2, 3, 4])
@pytest.mark.parametrize("W,H,D", [(1, 1, 1), (67, 13, 1), (130, 37, 7), (97, 21, 8), (97, 21, 9), (70, 30, 16),
                                   (129, 19, 31), (2369, 313, 8), (2369, 313, 16)])
def test_narrow_ncc(ctx, orc, radius, W, H, D):
    _check(ctx, orc, "ncc", radius, W, H, D)


@pytest.mark.parametrize("kind,radius", [("bt", 0), ("ssd", 1), ("ssd", 4), ("ncc", 1), ("ncc", 4)])
@pytest.mark.parametrize("W,H,D", [(90, 20, 79), (200, 9, 82), (333, 11, 144), (400, 7, 300)])
def test_filter_chunks(ctx, orc, kind, radius, W, H, D):
    _check(ctx, orc, kind, radius, W, H, D)


@pytest.mark.parametrize("kind,radius,D", [("bt", 0, 2300), ("ssd", 1, 2700), ("ssd", 1, 4500), ("ssd", 2, 2400),
                                           ("ssd", 4, 1300), ("ssd", 4, 2200), ("ncc", 1, 2000), ("ncc", 3, 1500),
                                           ("ncc", 4, 1100), ("ncc", 4, 1900)])
def test_wide(ctx, orc, kind, radius, D):
    _check(ctx, orc, kind, radius, D + 65, 3, D)
    if kind == "ssd":
        L, R = [torch.from_numpy(a).cuda() for a in _pair(D + 65, 3, D)]
        C = ctx.cost(L, R, D, kind="ssd", radius=radius)
        assert torch.equal(ctx.fast_wta(L, R, D, radius=radius)["disp"].view(torch.int16),
                           ctx.wta(C)["disp"].view(torch.int16))


@pytest.mark.parametrize("kind,radius,W,H,D", [
    # either side of the tile counts from which tiles are 8 rows high
    ("bt", 0, 641, 217, 16), ("bt", 0, 641, 222, 16), ("bt", 0, 641, 222, 17),
    ("ncc", 4, 641, 433, 8), ("ncc", 4, 641, 438, 8), ("ncc", 2, 641, 438, 9), ("ncc", 4, 1283, 459, 16),
    # the 3x3 of 16 lanes: two rows an item, then one
    ("ncc", 1, 641, 217, 20), ("ncc", 1, 641, 222, 20), ("ncc", 1, 1283, 565, 31), ("ncc", 2, 1283, 565, 31)])
def test_tile_counts(ctx, orc, kind, radius, W, H, D):
    _check(ctx, orc, kind, radius, W, H, D)
