"""Window costs and FastWTA at both tile heights (8 rows from 1480 tiles on, 4
below) and every lane count, bit-exact against the oracle; the filtered FastWTA
against filter, cost and winner in sequence."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

KIND_ID = {"bt": 0, "ssd": 1, "ncc": 2}


def _pair(W, H, seed):
    rng = np.random.default_rng(seed)
    L, R = [rng.random((H, W), dtype=np.float32) for _ in range(2)]
    L[:, : W // 5] = 0.5  # ties; the NCC of zero windows is NaN
    R[: H // 3, : W // 4] = 0.0
    return L, R


@pytest.mark.parametrize("kind,radius", [("bt", 0), ("ssd", 1), ("ssd", 4), ("ncc", 2)])
@pytest.mark.parametrize("W,H,D", [(2369, 313, 5), (2369, 313, 17), (1537, 481, 33), (130, 61, 40)])
def test_costs(ctx, orc, kind, radius, W, H, D):
    L, R = _pair(W, H, W + D)
    C = ctx.cost(torch.from_numpy(L).cuda(), torch.from_numpy(R).cuda(), D, kind=kind, radius=radius)
    ref = orc.cost_pair(L, R, D, KIND_ID[kind], radius, orc.LAYOUT_HWD)
    assert np.array_equal(C.cpu().numpy(), ref, equal_nan=True)


@pytest.mark.parametrize("radius", [1, 2, 3, 4])
@pytest.mark.parametrize("W,H,D", [(2369, 313, 7), (2369, 313, 40), (93, 38, 8), (77, 41, 9), (65, 33, 31),
                                   (65, 33, 32), (140, 9, 100), (3, 3, 64)])
def test_fast_wta(ctx, radius, W, H, D):
    L, R = [torch.from_numpy(a).cuda() for a in _pair(W, H, W + D + radius)]
    C = ctx.cost(L, R, D, kind="ssd", radius=radius)
    want = ctx.wta(C, norm=True)
    got = ctx.fast_wta(L, R, D, radius=radius, norm=True)
    for k in want:
        assert torch.equal(got[k].view(torch.int16 if k == "disp" else torch.int32),
                           want[k].view(torch.int16 if k == "disp" else torch.int32))
    for f in ("gauss5", "median7"):
        C, _ = ctx.cost_filtered(L, R, D, kind="ssd", radius=radius, prefilter=f)
        want = ctx.wta(C, norm=True)
        got = ctx.fast_wta_filtered(L, R, D, radius=radius, prefilter=f, norm=True)
        assert torch.equal(got["disp"].view(torch.int16), want["disp"].view(torch.int16))
        assert torch.equal(got["disp_norm"], want["disp_norm"])


def test_fast_wta_filtered_large_radius_and_bad_arguments(ctx):
    from thundervision_b200 import TdvError
    L, R = [torch.from_numpy(a).cuda() for a in _pair(60, 40, 1)]
    C, _ = ctx.cost_filtered(L, R, 12, kind="ssd", radius=6)
    got = ctx.fast_wta_filtered(L, R, 12, radius=6)["disp"]
    assert torch.equal(got.view(torch.int16), ctx.wta(C)["disp"].view(torch.int16))
    for bad in (dict(max_disp=0), dict(max_disp=12, radius=16)):
        with pytest.raises(TdvError):
            ctx.fast_wta_filtered(L, R, **bad)
