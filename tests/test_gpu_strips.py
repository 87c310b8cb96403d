"""Long strips over four paths, on both sides of the rule that sends D = 64 to
the accumulating passes: maps bit-exact against the oracle, and the path the
rule names."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sem,table", [("standard", "full"), ("ref_cpu", "ref"), ("ref_gpu", "ref")])
@pytest.mark.parametrize("W,H,lr,paths", [(4096, 9, 1, 4), (4095, 9, 1, 4), (4096, 9, None, 4), (4096, 9, 1, 8),
                                          (12288, 4, 1, 4)])
def test_strip(ctx, orc, sem, table, W, H, lr, paths):
    rng = np.random.default_rng(W + H)
    left = rng.integers(0, 256, size=(H, W)).astype(np.uint8)
    right = np.clip(np.roll(left, -7, 1).astype(int) + rng.integers(-9, 10, size=(H, W)), 0, 255).astype(np.uint8)
    l, r = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    out = []
    names = [n for n, _ in ctx.kernel_times(lambda: out.append(ctx.stereo_sgm(l, r, 64, 10, 120, paths=paths, lr=lr,
                                                                              semantics=sem, table=table)))]
    ctx.device_status()
    accumulates = paths == 4 and lr is not None and W >= (4096 if sem == "ref_cpu" else 12288)
    assert ("fused_sum_wta" in names) == (not accumulates)
    Lf, Rf = orc.u8_to_f32(left), orc.u8_to_f32(right)
    d, _, S = orc.sgm(orc.bt_cost(Lf, Rf, 64), Lf, 10, 120, paths=paths,
                      semantics={"standard": 0, "ref_cpu": 1, "ref_gpu": 2}[sem], table={"full": 0, "ref": 1}[table])
    if lr is not None:
        d, _ = orc.lr_check(S, d, thr=lr)
    np.testing.assert_array_equal(out[0]["disp"].cpu().numpy(), d)
