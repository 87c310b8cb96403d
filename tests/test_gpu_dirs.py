"""The fused path with every direction stored apart (kernels_dirs.cu) at the
edges of its lane classes, tiles and range rule, against the oracle (bit-exact:
integer arithmetic), against the accumulating fused passes, and with an
allocator that refuses its scratch."""
import numpy as np
import pytest
import torch

from thundervision_b200 import _lib as L
from thundervision_b200 import api
from thundervision_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def _oracle(orc, left, right, D, p1, p2, paths, sem, table, lr):
    Lf, Rf = orc.u8_to_f32(left), orc.u8_to_f32(right)
    C = orc.bt_cost(Lf, Rf, D)
    sems = {"standard": orc.SEM_STANDARD, "ref_cpu": orc.SEM_REF_CPU, "ref_gpu": orc.SEM_REF_GPU}
    tabs = {"full": orc.TABLE_FULL, "ref": orc.TABLE_REF}
    d, _, S = orc.sgm(C, Lf, p1, p2, paths=paths, semantics=sems[sem], table=tabs[table])
    if lr is None:
        return d, None
    return orc.lr_check(S, d, thr=lr)


def _check(ctx, orc, W, H, D, p1=10, p2=120, paths=8, sem="standard", table="full", lr=1, seed=0):
    rng = np.random.default_rng(seed + W * 7 + H * 3 + D)
    if seed % 2:  # runs of equal intensities: many ties
        left = np.repeat(rng.integers(0, 4, size=(H, (W + 2) // 3)) * 60, 3, 1)[:, :W].astype(np.uint8)
        right = np.roll(left, -min(3, W - 1), 1)
    else:
        left = rng.integers(0, 256, size=(H, W)).astype(np.uint8)
        right = np.clip(np.roll(left, -min(5, D - 1), 1).astype(int) + rng.integers(-9, 10, size=(H, W)), 0, 255)
        right = right.astype(np.uint8)
    out = ctx.stereo_sgm(torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda(), D, p1, p2, paths=paths,
                         semantics=sem, table=table, lr=lr, norm=True, right_disp=lr is not None)
    ctx.device_status()
    d, dr = _oracle(orc, left, right, D, p1, p2, paths, sem, table, lr)
    got = out["disp"].cpu().numpy()
    np.testing.assert_array_equal(got, d)
    want = np.where(got == 0xFFFF, np.float32(-1), got.astype(np.float32) / np.float32(D))
    np.testing.assert_array_equal(out["disp_norm"].cpu().numpy(), want)
    if lr is not None:
        np.testing.assert_array_equal(out["disp_right"].cpu().numpy(), dr)


SEMS = [("standard", "full"), ("ref_cpu", "ref"), ("ref_gpu", "ref")]


@pytest.mark.parametrize("sem,table", SEMS)
@pytest.mark.parametrize("W,H,D,paths,lr", [
    # lane classes and their edges; widths and heights at and off the tiles
    (47, 33, 16, 8, 1), (49, 48, 17, 4, 1), (24, 70, 32, 8, None), (97, 5, 33, 8, 0), (64, 64, 64, 8, 1),
    (129, 31, 65, 4, None), (70, 41, 128, 8, 1), (33, 90, 129, 8, 1), (261, 18, 256, 8, 1), (300, 37, 200, 4, 2),
    (12, 300, 8, 8, 1), (1, 40, 16, 8, 1), (40, 1, 40, 8, 1), (3, 2, 2, 8, 1), (31, 29, 250, 8, None),
])
def test_lane_classes(ctx, orc, sem, table, W, H, D, paths, lr):
    _check(ctx, orc, W, H, D, paths=paths, sem=sem, table=table, lr=lr, seed=(W + H) % 2)


@pytest.mark.parametrize("sem,table", SEMS)
@pytest.mark.parametrize("p1,p2", [(0, 0), (0.5, 127.5), (127.5, 127.5), (10, 128), (128, 20)])
def test_range_rule(ctx, orc, sem, table, p1, p2):
    """Penalties on both sides of the line between the byte and the 16-bit volumes."""
    for D in (24, 72):
        _check(ctx, orc, 90, 44, D, p1=p1, p2=p2, sem=sem, table=table, seed=1)
        _check(ctx, orc, 90, 44, D, p1=p1, p2=p2, sem=sem, table=table, seed=2)


@pytest.mark.parametrize("sem,table", SEMS)
def test_two_lines_per_lane_group(ctx, orc, sem, table):
    """Wide enough for two lines per lane group (D > 128), odd sizes."""
    _check(ctx, orc, 1205, 61, 136, sem=sem, table=table, seed=2)


@pytest.mark.parametrize("p2,paths", [(120, 8), (120, 4), (128, 8), (300.5, 4)])
def test_batch_on_both_sides_of_the_range_rule(ctx, p2, paths):
    """Batches store the directions apart up to P2 = 127.5 and accumulate above;
    both equal the per-pair calls."""
    pairs = []
    for i, (W, H, D, lr) in enumerate([(70, 40, 12, 1), (333, 61, 32, None), (96, 130, 64, 2), (240, 33, 100, None),
                                       (501, 29, 200, 1), (5, 3, 8, 1)]):
        left, right, _, _ = syn.make_pair(max(W, 40), max(H, 30), D, 40 + i, n_rects=3)
        cut = lambda a: torch.from_numpy(np.ascontiguousarray(a[:H, :W])).cuda()
        pairs.append((cut(left), cut(right), D, lr))
    b = api.Batch(ctx, pairs, 10, p2, paths=paths, norm=True, right_disp="lr")
    for _ in range(2):
        out = b.run()
        b.status()
        for (lt, rt, D, lr), o in zip(pairs, out):
            want = ctx.stereo_sgm(lt, rt, D, 10, p2, paths=paths, lr=lr, norm=True, right_disp=lr is not None)
            for k in want:
                assert torch.equal(o[k].view(torch.int32 if k == "disp_norm" else torch.int16),
                                   want[k].view(torch.int32 if k == "disp_norm" else torch.int16))
    b.close()


@pytest.mark.slow
def test_batch_waves(ctx):
    """Three full-HD pairs at D = 256 and a small one: more volumes than one wave holds."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    pairs = []
    for W, H, D in [(1920, 1080, 256), (1920, 1080, 256), (64, 48, 32), (1920, 1080, 200)]:
        left = torch.randint(0, 256, (H, W), generator=g, device="cuda", dtype=torch.uint8)
        pairs.append((left, torch.roll(left, -9, 1), D, 1))
    b = api.Batch(ctx, pairs, 10, 120)
    for order in (0, 1):
        b.set_tiles(order=order)
        out = b.run()
        b.status()
        for (lt, rt, D, lr), o in zip(pairs, out):
            want = ctx.stereo_sgm(lt, rt, D, 10, 120, lr=lr)["disp"]
            assert torch.equal(o["disp"].view(torch.int16), want.view(torch.int16))
    b.close()


def test_refused_scratch_falls_back():
    """An allocator without room for the directions' volumes: the calls run the
    accumulating passes, with the same maps."""
    W, H, D = 320, 200, 64
    left, right, _, _ = syn.make_pair(W, H, D, 5, n_rects=6)
    lt, rt = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    limit = 2 * W * H * D + (1 << 20)  # one 16-bit volume fits, eight of bytes do not
    live, refused = {}, []

    def alloc(n, user):
        if n > limit:
            refused.append(n)
            return None
        t = torch.empty(n, dtype=torch.uint8, device="cuda")
        live[t.data_ptr()] = t
        return t.data_ptr()

    def release(p, user):
        live.pop(p, None)

    small, big = api.Context(0), api.Context(0)
    try:
        small.set_allocator(alloc, release)
        small.reserve(W, H, D)
        for _ in range(2):
            a = small.stereo_sgm(lt, rt, D, 10, 120, lr=1, semantics="ref_cpu", table="ref")
            f = small.stereo_sgm_frames([lt, rt], [rt, lt], D, 10, 120, lr=1)
        b = big.stereo_sgm(lt, rt, D, 10, 120, lr=1, semantics="ref_cpu", table="ref")
        g = big.stereo_sgm_frames([lt, rt], [rt, lt], D, 10, 120, lr=1)
        small.device_status()
        assert len(refused) <= 2
        assert torch.equal(a["disp"].to(torch.int32), b["disp"].to(torch.int32))
        for x, y in zip(f, g):
            assert torch.equal(x["disp"].to(torch.int32), y["disp"].to(torch.int32))
    finally:
        small.close()
        big.close()


def test_captured_call(ctx):
    """One call captured and replayed on new inputs equals direct calls."""
    W, H, D = 256, 96, 48
    rng = np.random.default_rng(0)
    pairs = [torch.from_numpy(rng.integers(0, 256, size=(2, H, W)).astype(np.uint8)).cuda() for _ in range(2)]
    buf = pairs[0].clone()
    c = api.Context(0)
    try:
        c.stereo_sgm(buf[0], buf[1], D, 10, 120, lr=1)
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(s), torch.cuda.graph(g, stream=s):
            out = c.stereo_sgm(buf[0], buf[1], D, 10, 120, lr=1)
        for p in (pairs[1], pairs[0]):
            buf.copy_(p)
            g.replay()
            want = ctx.stereo_sgm(p[0], p[1], D, 10, 120, lr=1)["disp"]
            torch.cuda.synchronize()
            assert torch.equal(out["disp"].to(torch.int32), want.to(torch.int32))
    finally:
        g = None
        c.close()
