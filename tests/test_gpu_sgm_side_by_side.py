"""The general aggregation with its passes side by side (kernels_sgm_dirs.cu)
against the oracle, bit-exact: the additions are the reference's, in its order.
Disparity ranges at and off the lane groups and the 32-byte accesses, both
layouts, every recurrence and table, a volume that does not start on 32 bytes,
16-bit costs, and allocators that leave room for two volumes, or for none."""
import numpy as np
import pytest
import torch

from thundervision_b200 import api

pytestmark = pytest.mark.gpu

SEMS = {"standard": 0, "ref_cpu": 1, "ref_gpu": 2}
TABS = {"full": 0, "ref": 1}


def _volume(rng, H, W, D):
    C = rng.uniform(0, 3, size=(H, W, D)).astype(np.float32)
    for x in range(min(W, D)):
        C[:, x, x + 1:] = np.inf
    C[rng.random(C.shape) < 0.002] = np.nan
    C[:, :, : D // 2][rng.random((H, W, D // 2)) < 0.2] = 0.5  # ties
    return C


def _run(ctx, orc, C, guide, p1, p2, paths, sem, table, p2_mode, layout="hwd", offset=0, lr=1):
    H, W, D = C.shape
    d, _, S = orc.sgm(C, guide, p1, p2, p2_mode=1 if p2_mode == "adjust" else 0, paths=paths, table=TABS[table],
                      semantics=SEMS[sem])
    dl, dr = orc.lr_check(S, d, thr=lr)
    Ct = torch.from_numpy(C if layout == "hwd" else np.ascontiguousarray(C.transpose(1, 0, 2))).cuda()
    buf = torch.empty(C.size + offset, dtype=torch.float32, device="cuda")
    vol = buf[offset:].view(Ct.shape)
    vol.copy_(Ct)
    agg = torch.empty(Ct.shape, device="cuda")
    g = torch.from_numpy(guide).cuda()
    out = ctx.sgm(vol, p1, p2, guide=g, p2_mode=p2_mode, paths=paths, table=table, semantics=sem, layout=layout,
                  aggreg=agg)
    got = agg.cpu().numpy()
    np.testing.assert_array_equal(got if layout == "hwd" else got.transpose(1, 0, 2), S)
    np.testing.assert_array_equal(out["disp"].cpu().numpy(), d)
    out = ctx.sgm(vol, p1, p2, guide=g, p2_mode=p2_mode, paths=paths, table=table, semantics=sem, layout=layout,
                  lr=lr, right=True)
    np.testing.assert_array_equal(out["disp"].cpu().numpy(), dl)
    np.testing.assert_array_equal(out["disp_right"].cpu().numpy(), dr)


CASES = [(23, 17, 8, "hwd", 0), (17, 23, 31, "ref", 0), (40, 9, 32, "hwd", 1), (9, 40, 33, "hwd", 0),
         (30, 21, 64, "ref", 0), (21, 30, 65, "hwd", 0), (26, 14, 100, "hwd", 0), (14, 26, 128, "ref", 3),
         (19, 8, 136, "hwd", 0), (8, 19, 256, "hwd", 0), (1, 12, 16, "hwd", 0), (12, 1, 16, "ref", 0),
         (70, 66, 24, "hwd", 0)]


@pytest.mark.parametrize("sem,table", [("standard", "full"), ("ref_cpu", "ref"), ("ref_gpu", "ref"),
                                       ("ref_cpu", "full")])
@pytest.mark.parametrize("W,H,D,layout,offset", CASES)
def test_matches_oracle(ctx, orc, sem, table, W, H, D, layout, offset):
    rng = np.random.default_rng(W * 31 + H * 7 + D)
    C = _volume(rng, H, W, D)
    guide = rng.integers(0, 5, size=(H, W)).astype(np.float32) / 4
    _run(ctx, orc, C, guide, 0.3, 1.7, 8, sem, table, "adjust" if (W + D) % 2 else "const", layout, offset)
    _run(ctx, orc, C, guide, 0.3, 1.7, 4, sem, table, "const" if (W + D) % 2 else "adjust", layout, offset)


@pytest.mark.parametrize("room", [2, 0])
@pytest.mark.parametrize("sem,table", [("standard", "full"), ("ref_cpu", "ref"), ("ref_gpu", "ref")])
def test_refused_volumes(orc, room, sem, table):
    W, H, D = 61, 43, 40
    vol = (W * H * D * 4 + 255) // 256 * 256
    live = {}

    def alloc(n, user):
        if n > max(room, 1) * vol or (room == 0 and n == 2 * vol):
            return None
        t = torch.empty(n, dtype=torch.uint8, device="cuda")
        live[t.data_ptr()] = t
        return t.data_ptr()

    def release(p, user):
        live.pop(p, None)

    ctx = api.Context(0)
    try:
        ctx.set_allocator(alloc, release)
        rng = np.random.default_rng(3)
        C = _volume(rng, H, W, D)
        guide = rng.integers(0, 5, size=(H, W)).astype(np.float32) / 4
        for _ in range(2):
            _run(ctx, orc, C, guide, 0.3, 1.7, 8, sem, table, "adjust")
    finally:
        ctx.close()


def test_u16_cost_equals_float(ctx):
    rng = np.random.default_rng(5)
    for D in (24, 30, 200):
        left, right = [torch.from_numpy(rng.integers(0, 256, size=(37, 90)).astype(np.uint8)).cuda() for _ in range(2)]
        a = ctx.sgm(ctx.cost(left, right, D), 10, 120.25, lr=1, table="ref", semantics="ref_cpu")
        b = ctx.sgm(ctx.cost(left, right, D, dtype="u16"), 10, 120.25, lr=1, table="ref", semantics="ref_cpu")
        assert torch.equal(a["disp"].to(torch.int32), b["disp"].to(torch.int32))
