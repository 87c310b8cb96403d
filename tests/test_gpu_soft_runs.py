"""The soft SGM's load rings and whole-vector accesses where they can go wrong:
disparity ranges at and off the vector widths, walks shorter and longer than
the ring, segments that do not divide a walk, and a cost volume that does not
start on 16 bytes (which takes the scalar accesses).

Costs and penalties are multiples of 1/8, so every path cost is exact in FP32
and both precisions route the gradient alike.  FP64 against the FP64 oracle:
dhat 1e-12, gradients 1e-9 (sums over disparities are reduced in another
order); FP32: 1e-4 norm-wise, the bar the path is held to.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("W,H,D,paths,ck", [
    (9, 5, 1, 8, 0), (6, 10, 31, 8, 4), (8, 3, 32, 4, 3), (5, 12, 36, 8, 0), (11, 7, 62, 8, 5), (13, 6, 64, 8, 32),
    (6, 9, 100, 8, 4), (7, 5, 102, 4, 2), (1, 9, 128, 8, 3), (9, 1, 128, 8, 0), (5, 6, 200, 8, 1), (6, 5, 250, 8, 3),
    (70, 4, 256, 4, 32),
])
def test_runs_match_oracle(ctx, orc, W, H, D, paths, ck, offset):
    from thundervision_b200.soft import soft_sgm
    rng = np.random.default_rng(W * 1000 + H * 100 + D)
    C = rng.integers(0, 40 * 8, size=(H, W, D)) / 8.0
    g = rng.normal(size=(H, W))
    p1, p2, tau = 1.5, 7.25, 2.0
    _, dh_ref = orc.soft_sgm_fwd(C, p1, p2, tau=tau, paths=paths)
    dC_ref, d1_ref, d2_ref = orc.soft_sgm_bwd(C, p1, p2, g, tau=tau, paths=paths)
    for dt in (torch.float64, torch.float32):
        buf = torch.empty(C.size + offset, dtype=dt, device="cuda")
        c = buf[offset:].view(H, W, D)
        c.copy_(torch.from_numpy(C))
        c = c.detach().requires_grad_(True)
        pen = torch.tensor([p1, p2], dtype=dt, device="cuda", requires_grad=True)
        dh = soft_sgm(c, pen[0], pen[1], tau=tau, paths=paths, checkpoint=ck, ctx=ctx)
        (dh * torch.tensor(g, dtype=dt, device="cuda")).sum().backward()
        got, gp = c.grad.double().cpu().numpy(), pen.grad.double().cpu().numpy()
        dh = dh.detach().double().cpu().numpy()
        if dt == torch.float64:
            np.testing.assert_allclose(dh, dh_ref, rtol=1e-12, atol=1e-12)
            np.testing.assert_allclose(got, dC_ref, rtol=1e-9, atol=1e-11)
            np.testing.assert_allclose(gp, [d1_ref, d2_ref], rtol=1e-9, atol=1e-11)
        else:
            np.testing.assert_allclose(dh, dh_ref, rtol=1e-4, atol=1e-4)
            assert np.linalg.norm(got - dC_ref) <= 1e-4 * max(np.linalg.norm(dC_ref), 1e-3)
            scale = max(abs(d1_ref), abs(d2_ref), 1e-3 * np.abs(g).sum())
            assert np.abs(gp - [d1_ref, d2_ref]).max() <= 1e-4 * scale
