"""The work a user of this library has it do, as measurable cases.

Every case goes through the Python front end (thundervision_b200.api, .soft
and .reconstruction) on device tensors.  A case is a dict; its "kind" names
the call:

  fused   Context.stereo_sgm: one uint8 pair, Birchfield-Tomasi + SGM + WTA
  frames  Context.stereo_sgm_frames: a short sequence of equal-size pairs
  batch   Batch.run: pairs of uneven size and disparity range
  sgm     Context.cost (BT, the reference's DSI layout) + Context.sgm on a
          float pair in [0, 1] with the reference's penalties (30/255,
          150/255 over the intensity step): the drop-in stage chain
  agg     Context.sgm of a float DSI with the aggregated volume kept, then
          Context.subpixel: the refinement that needs the volume
  recon   Reconstruction.update: color frames to a reprojected mesh
  dp      Context.cost + Context.dp: the scanline matcher on a window cost
  fwta    Context.fast_wta: window SSD + WTA without a DSI
  soft    soft.soft_sgm forward and backward: a differentiable matcher's
          training step on a cost volume

Inputs are textured stereo pairs (blurred noise, a slanted plane and
rectangles at constant disparity, sensor noise, 2 % salt and pepper), made on
the device from the seed.
"""
import math

import numpy as np
import torch

from thundervision_b200 import api, reconstruction
from thundervision_b200.soft import soft_sgm


def listed():
    return [
        # a thumbnail-sized preview pair: launches and latency are all there is
        {"name": "pair_384x288_d16", "kind": "fused", "W": 384, "H": 288, "D": 16, "paths": 8,
         "semantics": "standard", "table": "full", "lr": 1},
        # an ordinary camera pair
        {"name": "pair_640x480_d64", "kind": "fused", "W": 640, "H": 480, "D": 64, "paths": 8,
         "semantics": "standard", "table": "full", "lr": 1},
        # a cropped region of interest: odd size, odd disparity range, four
        # paths for speed, no left-right check
        {"name": "pair_1003x701_d100_4path", "kind": "fused", "W": 1003, "H": 701, "D": 100, "paths": 4,
         "semantics": "standard", "table": "full", "lr": -1},
        # a full-HD pair under the reference's CPU recurrence and path table
        {"name": "pair_1920x1080_d256_ref", "kind": "fused", "W": 1920, "H": 1080, "D": 256, "paths": 8,
         "semantics": "ref_cpu", "table": "ref", "lr": 1},
        # a stretch of full-HD video
        {"name": "frames_1920x1080_d256", "kind": "frames", "W": 1920, "H": 1080, "D": 256, "paths": 8,
         "semantics": "standard", "table": "full", "lr": 1, "n": 4},
        # an image collection matched in one go
        {"name": "batch_16", "kind": "batch", "n": 16, "shapes": 7, "wmax": 1920, "hmax": 1080, "dmax": 256,
         "paths": 8, "lr": 1},
        # the reference's stage chain, small and full HD
        {"name": "sgm_640x480_d64", "kind": "sgm", "W": 640, "H": 480, "D": 64, "lr": 1},
        {"name": "sgm_1920x1080_d128", "kind": "sgm", "W": 1920, "H": 1080, "D": 128, "lr": -1},
        # a float window-cost DSI aggregated, the volume kept for refinement
        {"name": "agg_640x480_d64", "kind": "agg", "W": 640, "H": 480, "D": 64, "cost": "ssd", "radius": 2,
         "paths": 8},
        # the reconstruction chain as its factory configures it (SSD 7x7, WTA)
        {"name": "recon_1920x1080_d64", "kind": "recon", "W": 1920, "H": 1080, "D": 64},
        # the scanline matcher on the NCC cost
        {"name": "dp_640x480_d64_ncc", "kind": "dp", "W": 640, "H": 480, "D": 64, "cost": "ncc", "radius": 4},
        # a training step through the aggregation
        {"name": "soft_960x540_d128", "kind": "soft", "W": 960, "H": 540, "D": 128, "paths": 8,
         "checkpoint": 32},
    ]


# ------------------------------------------------------------------- drawing
def _logint(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["fused", "fused", "fused", "frames", "batch", "sgm", "agg", "recon", "dp", "fwta", "soft"])
    W = _logint(rng, 160, 1920)
    H = max(96, min(1080, int(round(W * rng.uniform(0.45, 0.8)))))
    if rng.random() < 0.15:
        W, H = H, W  # portrait
    W = max(96, min(W, 1920))
    c = {"kind": kind, "W": W, "H": H}
    # disparity ranges: mostly the usual powers of two, odd ones among them
    D = rng.choice([16, 32, 64, 128, 256]) if rng.random() < 0.6 else _logint(rng, 9, 256)
    lr = rng.choice([-1, 1, 1])
    sem, table = rng.choice([("standard", "full"), ("standard", "full"), ("ref_cpu", "ref"), ("ref_gpu", "ref")])
    if kind == "fused":
        c.update(D=D, paths=rng.choice([4, 8, 8]), semantics=sem, table=table, lr=lr)
    elif kind == "frames":
        c.update(D=D, paths=rng.choice([4, 8, 8]), semantics=sem, table=table, lr=lr, n=rng.randint(2, 4))
    elif kind == "batch":
        del c["W"], c["H"]
        c.update(n=rng.randint(3, 12), shapes=rng.randrange(1 << 20), wmax=_logint(rng, 400, 1600),
                 hmax=_logint(rng, 300, 900), dmax=rng.choice([64, 128, 256]), paths=rng.choice([4, 8]), lr=lr)
    elif kind == "sgm":
        c.update(D=min(D, 128), lr=lr)
    elif kind == "agg":
        c.update(D=min(D, 128), cost=rng.choice(["bt", "ssd", "ncc"]), radius=rng.randint(1, 4),
                 paths=rng.choice([4, 8]))
        c["W"], c["H"] = min(c["W"], 1000), min(c["H"], 700)
    elif kind == "recon":
        c.update(D=rng.choice([32, 64, 64, 100]))
    elif kind == "dp":
        c.update(D=min(D, 128), cost=rng.choice(["bt", "ssd", "ncc"]), radius=rng.randint(1, 4))
    elif kind == "fwta":
        c.update(D=min(D, 128), radius=rng.randint(1, 4))
    else:
        c.update(D=min(D, 128), paths=rng.choice([4, 8]), checkpoint=rng.choice([0, 16, 32]))
        c["W"], c["H"] = min(c["W"], 960), min(c["H"], 640)
    return c


# -------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _texture(g, H, W):
    """Uniform noise blurred with a Gaussian (sigma 1.5), rescaled to 0..255."""
    r, s = 5, 1.5
    k = [math.exp(-0.5 * (i / s) ** 2) for i in range(-r, r + 1)]
    n = torch.rand((H + 2 * r, W + 2 * r), generator=g, device="cuda")
    t = sum(w * n[:, i:i + W] for i, w in enumerate(k))
    t = sum(w * t[i:i + H, :] for i, w in enumerate(k))
    lo, hi = t.min(), t.max()
    return (t - lo) * (255.0 / (hi - lo))


def _scene(W, H, D, seed):
    """(left, right) float textures in 0..255 before noise, and the left
    view's disparity field (int64)."""
    g = _gen(seed)
    rng = np.random.default_rng(seed)
    right = _texture(g, H, W)
    d = torch.full((H, W), min(2, D - 1), dtype=torch.int64, device="cuda")
    x = torch.arange(W, device="cuda")
    plane = torch.round((0.1 + 0.5 * x / max(W - 1, 1)) * (D - 1)).long()
    d[H // 4:H // 4 + H // 2, W // 5:W // 5 + W // 2] = plane[W // 5:W // 5 + W // 2]
    for _ in range(8):
        rw, rh = int(rng.integers(W // 12, W // 4)), int(rng.integers(H // 12, H // 4))
        x0, y0 = int(rng.integers(0, W - rw)), int(rng.integers(0, H - rh))
        d[y0:y0 + rh, x0:x0 + rw] = int(rng.integers(0, D))
    src = x.view(1, W) - d
    fresh = torch.rand((H, W), generator=g, device="cuda") * 255.0
    left = torch.where(src >= 0, right.gather(1, src.clamp(min=0)), fresh)
    return left, right, d, g


def _sensor(img, g):
    """Sensor noise (sigma 2), 2 % salt and pepper, 8-bit."""
    img = img + 2.0 * torch.randn(img.shape, generator=g, device="cuda")
    hit = torch.rand(img.shape, generator=g, device="cuda")
    img = torch.where(hit < 0.01, torch.zeros_like(img), torch.where(hit > 0.99, torch.full_like(img, 255.0), img))
    return img.round().clamp(0, 255).to(torch.uint8)


def _pair(W, H, D, seed):
    left, right, d, g = _scene(W, H, D, seed)
    return _sensor(left, g), _sensor(right, g), d


def _unit_pair(W, H, D, seed):
    left, right, d = _pair(W, H, D, seed)
    return left.float() / 255.0, right.float() / 255.0, d


def _batch_shapes(c):
    rng = np.random.default_rng(c["shapes"])
    out = []
    for _ in range(c["n"]):
        W = 16 * int(rng.integers(20, c["wmax"] // 16 + 1))
        H = 16 * int(rng.integers(15, max(16, c["hmax"] // 16) + 1))
        out.append((W, H, int(rng.choice([d for d in (32, 64, 128, 256) if d <= c["dmax"]]))))
    return out


def _camera(W, H, sign):
    """A mildly distorted camera turned by a fraction of a degree."""
    a = sign * 0.004
    K = [[0.9 * W, 0, W / 2 - 3.5], [0, 0.9 * W, H / 2 + 2.25], [0, 0, 1]]
    R = [[math.cos(a), 0, math.sin(a)], [0, 1, 0], [-math.sin(a), 0, math.cos(a)]]
    P = [[0.88 * W, 0, W / 2], [0, 0.88 * W, H / 2], [0, 0, 1]]
    return reconstruction.Camera(K, [-0.12, 0.03, 1e-4, -2e-4, 0.0], R, P)


def prepare(case, seed):
    k = case["kind"]
    lr = case.get("lr", -1)
    s = {"case": case, "lr": None if lr < 0 else lr, "ctx": api.default_context()}
    if k == "fused":
        s["left"], s["right"], _ = _pair(case["W"], case["H"], case["D"], seed)
    elif k == "frames":
        p = [_pair(case["W"], case["H"], case["D"], seed * 8 + i) for i in range(case["n"])]
        s["left"], s["right"] = [q[0] for q in p], [q[1] for q in p]
    elif k == "batch":
        pairs = []
        for i, (W, H, D) in enumerate(_batch_shapes(case)):
            left, right, _ = _pair(W, H, D, seed * 64 + i)
            pairs.append((left, right, D))
        s["batch"] = api.Batch(s["ctx"], pairs, 10, 120, paths=case["paths"], lr=s["lr"], norm=True)
    elif k == "recon":
        W, H = case["W"], case["H"]
        left, right, _, g = _scene(W, H, case["D"], seed)
        tint = torch.tensor([0.8, 1.0, 0.9], device="cuda")
        s["left"] = _sensor(left.unsqueeze(2) * tint, g)
        s["right"] = _sensor(right.unsqueeze(2) * tint, g)
        s["ctx"] = api.Context()  # a captured chain keeps its context's scratch
        m = reconstruction.StereoMatcher(s["ctx"], case["D"], "ssd", "wta")
        q = [1, 0, 0, -W / 2, 0, 1, 0, -H / 2, 0, 0, 0, 0.9 * W, 0, 0, 4.0, 0.5]
        s["recon"] = reconstruction.Reconstruction(s["ctx"], W, H, _camera(W, H, 1), _camera(W, H, -1), Q=q,
                                                   matcher=m)
    elif k == "soft":
        left, right, d = _pair(case["W"], case["H"], case["D"], seed)
        cost = s["ctx"].cost(left, right, case["D"])
        # cells left of the image: the largest Birchfield-Tomasi cost
        s["cost"] = cost.clamp_(max=255.0).requires_grad_(True)
        s["pen"] = torch.tensor([10.0, 120.0], device="cuda", requires_grad=True)
        s["gt"] = d.float()
    else:
        s["left"], s["right"], _ = _unit_pair(case["W"], case["H"], case["D"], seed)
        if k == "agg":
            s["dsi"] = s["ctx"].cost(s["left"], s["right"], case["D"], kind=case["cost"], radius=case["radius"])
            s["S"] = torch.empty_like(s["dsi"])
    return s


def run(s):
    c, ctx, k = s["case"], s["ctx"], s["case"]["kind"]
    if k == "fused":
        return ctx.stereo_sgm(s["left"], s["right"], c["D"], 10, 120, paths=c["paths"], table=c["table"],
                              semantics=c["semantics"], lr=s["lr"], norm=True, right_disp=s["lr"] is not None)
    if k == "frames":
        return ctx.stereo_sgm_frames(s["left"], s["right"], c["D"], 10, 120, paths=c["paths"], table=c["table"],
                                     semantics=c["semantics"], lr=s["lr"], right_disp=s["lr"] is not None)
    if k == "batch":
        return s["batch"].run()
    if k == "sgm":
        C = ctx.cost(s["left"], s["right"], c["D"], layout="ref")
        out = ctx.sgm(C, 30.0 / 255.0, 150.0 / 255.0, guide=s["left"], p2_mode="adjust", table="ref",
                      semantics="ref_gpu", layout="ref", lr=s["lr"], norm=True)
        out["dsi"] = C
        return out
    if k == "agg":
        out = ctx.sgm(s["dsi"], 0.05, 0.7, paths=c["paths"], aggreg=s["S"])
        out["S"] = s["S"]
        out["subpixel"] = ctx.subpixel(s["S"], out["disp"])
        return out
    if k == "recon":
        return s["recon"].update(s["left"], s["right"])
    if k == "dp":
        C = ctx.cost(s["left"], s["right"], c["D"], kind=c["cost"], radius=0 if c["cost"] == "bt" else c["radius"])
        out = ctx.dp(C, norm=True)
        out["dsi"] = C
        return out
    if k == "fwta":
        return ctx.fast_wta(s["left"], s["right"], c["D"], radius=c["radius"], norm=True)
    dhat = soft_sgm(s["cost"], s["pen"][0], s["pen"][1], tau=1.0, paths=c["paths"], checkpoint=c["checkpoint"],
                    ctx=ctx)
    loss = torch.nn.functional.smooth_l1_loss(dhat, s["gt"])
    dcost, dpen = torch.autograd.grad(loss, (s["cost"], s["pen"]))
    return {"dhat": dhat.detach(), "dcost": dcost, "dpen": dpen}


# ---------------------------------------------------------------------- work
def work(case):
    """Bytes: inputs read once, outputs written once.  Operations: per cell
    (pixel x disparity) and path 8 for the recurrence, 9 for Birchfield-Tomasi
    and 3 per window tap, 1 per cell for the winner-take-all."""
    k = case["kind"]
    if k == "batch":
        b = f = 0
        for W, H, D in _batch_shapes(case):
            b += W * H * (2 + 6)
            f += W * H * D * (10 + 8 * case["paths"])
        return {"bytes": b, "flops": f}
    W, H, D = case["W"], case["H"], case["D"]
    n, cells = W * H, W * H * D
    taps = 3 * (2 * case.get("radius", 3) + 1) ** 2 if case.get("cost", "ssd") != "bt" else 9
    if k == "fused":
        return {"bytes": n * (2 + 6 + (2 if case["lr"] >= 0 else 0)), "flops": cells * (10 + 8 * case["paths"])}
    if k == "frames":
        return {"bytes": case["n"] * n * (2 + 2 + (2 if case["lr"] >= 0 else 0)),
                "flops": case["n"] * cells * (10 + 8 * case["paths"])}
    if k == "sgm":
        return {"bytes": n * (8 + 6) + 4 * cells, "flops": cells * (10 + 8 * 8)}
    if k == "agg":
        return {"bytes": 8 * cells + n * 6, "flops": cells * (1 + 8 * case["paths"])}
    if k == "recon":
        return {"bytes": n * (6 + 3 + 4 + 24), "flops": cells * (3 * 49 + 1)}
    if k == "dp":
        return {"bytes": n * (8 + 6) + 4 * cells, "flops": cells * (taps + 4)}
    if k == "fwta":
        return {"bytes": n * (8 + 6), "flops": cells * taps}
    return {"bytes": 8 * cells + 8 * n, "flops": cells * (2 * 8 * case["paths"] + 12)}


# --------------------------------------------------------------------- exact
def _clamped(im, dx, dy):
    """im shifted so that [y, x] is im[y + dy, x + dx], clamped to the edge."""
    H, W = im.shape
    y = (torch.arange(H, device=im.device) + dy).clamp(0, H - 1)
    x = (torch.arange(W, device=im.device) + dx).clamp(0, W - 1)
    return im[y][:, x]


def _dsi64(left, right, D, kind, r):
    """The (H, W, D) matching cost in 64 bits; +inf where x - d < 0."""
    L, R = left.double(), right.double()
    H, W = L.shape
    out = torch.full((H, W, D), math.inf, dtype=torch.float64, device=L.device)

    def half(im):
        a, b = 0.5 * (im + _clamped(im, -1, 0)), 0.5 * (im + _clamped(im, 1, 0))
        return torch.minimum(im, torch.minimum(a, b)), torch.maximum(im, torch.maximum(a, b))

    if kind == "bt":
        (ln, lx), (rn, rx) = half(L), half(R)
    win = range(-r, r + 1)
    for d in range(min(D, W)):
        if kind == "bt":
            l, n, x = L[:, d:], ln[:, d:], lx[:, d:]
            rr, rrn, rrx = R[:, :W - d], rn[:, :W - d], rx[:, :W - d]
            a = torch.maximum(l - rrx, rrn - l).clamp(min=0)
            b = torch.maximum(rr - x, n - rr).clamp(min=0)
            v = torch.minimum(a, b)
        else:
            v = ls = rs = 0.0
            for j in win:
                for i in win:
                    lv, rv = _clamped(L, i, j)[:, d:], _clamped(R, i - d, j)[:, d:]
                    if kind == "ssd":
                        v = v + (lv - rv) ** 2
                    else:
                        v, ls, rs = v + lv * rv, ls + lv * lv, rs + rv * rv
            if kind == "ncc":
                v = 1.0 - v / torch.sqrt(ls * rs)
        out[:, d:, d] = v
    return out


_DIRS = [(1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (-1, -1), (-1, 1), (1, -1)]


def _steps(W, H, dx, dy):
    """The cells of one direction in walk order, step by step: (pixel indices,
    previous pixels' indices) with -1 where the path starts."""
    dev = "cuda"
    if dy == 0:
        ys = torch.arange(H, device=dev)
        for t in range(W):
            x = t if dx > 0 else W - 1 - t
            yield ys * W + x, (ys * W + x - dx if t else torch.full_like(ys, -1))
        return
    xs = torch.arange(W, device=dev)
    for t in range(H):
        y = t if dy > 0 else H - 1 - t
        px = xs - dx
        prev = torch.where((px >= 0) & (px < W), (y - dy) * W + px, torch.full_like(xs, -1))
        yield y * W + xs, (prev if t else torch.full_like(xs, -1))


def _walk64(C, p1, p2, dx, dy, W, H, codes=None, kstar=None):
    """L of one direction over the flat (H*W, D) cost; optionally the branch
    every cell's minimum took (same disparity, d-1, d+1, jump; the first that
    attains it) and the lowest argmin of every pixel."""
    L = torch.empty_like(C)
    for cur, prev in _steps(W, H, dx, dy):
        P = L[prev.clamp(min=0)]
        m = P.min(1, keepdim=True).values
        inf = torch.full_like(m, math.inf)
        b = torch.cat([inf, P[:, :-1]], 1) + p1
        e = torch.cat([P[:, 1:], inf], 1) + p1
        j = (m + p2).expand_as(P)
        mn = torch.minimum(torch.minimum(P, b), torch.minimum(e, j))
        start = (prev < 0).unsqueeze(1)
        L[cur] = torch.where(start, C[cur], C[cur] + mn - m)
        if codes is not None:
            code = torch.full_like(P, 3, dtype=torch.uint8)
            code[e == mn] = 2
            code[b == mn] = 1
            code[P == mn] = 0
            codes[cur] = code
            kstar[cur] = L[cur].argmin(1)
    return L


def _back64(dS, codes, kstar, dx, dy, W, H):
    """dC of one direction's L, and the sums that reach P1 and P2."""
    G = dS.clone()
    g1 = g2 = 0.0
    for cur, prev in reversed(list(_steps(W, H, dx, dy))):
        ok = prev >= 0
        if not bool(ok.any()):
            continue
        g, c, p = G[cur[ok]], codes[cur[ok]], prev[ok]
        z = torch.zeros_like(g)
        same, up, dn, jump = (torch.where(c == v, g, z) for v in range(4))
        back = same
        back[:, :-1] += up[:, 1:]
        back[:, 1:] += dn[:, :-1]
        j = jump.sum(1)
        back.scatter_add_(1, kstar[p].unsqueeze(1), (j - g.sum(1)).unsqueeze(1))
        G[p] += back
        g1 = g1 + up.sum() + dn.sum()
        g2 = g2 + j.sum()
    return G, g1, g2


def _exact_soft(case, seed):
    W, H, D = case["W"], case["H"], case["D"]
    left, right, d = _pair(W, H, D, seed)
    C = _dsi64(left, right, D, "bt", 0).clamp(max=255.0).view(H * W, D)
    dirs = _DIRS[:case["paths"]]
    S = torch.zeros_like(C)
    tape = []
    for dx, dy in dirs:
        codes = torch.empty(C.shape, dtype=torch.uint8, device="cuda")
        kstar = torch.empty(H * W, dtype=torch.int64, device="cuda")
        S += _walk64(C, 10.0, 120.0, dx, dy, W, H, codes, kstar)
        tape.append((codes, kstar))
    S.requires_grad_(True)
    ds = torch.arange(D, dtype=torch.float64, device="cuda")
    dhat = (torch.softmax(-S, 1) * ds).sum(1).view(H, W)
    loss = torch.nn.functional.smooth_l1_loss(dhat, d.double())
    dS, = torch.autograd.grad(loss, S)
    dC, g1, g2 = torch.zeros_like(C), 0.0, 0.0
    for (dx, dy), (codes, kstar) in zip(dirs, tape):
        G, a, b = _back64(dS, codes, kstar, dx, dy, W, H)
        dC += G
        g1, g2 = g1 + a, g2 + b
    return {"dhat": dhat.detach(), "dcost": dC.view(H, W, D), "dpen": torch.stack([g1, g2])}


def exact(case, seed):
    """64-bit values of the computed outputs.  Disparity maps (and d/D of
    them, and what is measured from them) are whole numbers chosen by the
    smallest cost and have none; the image chain's outputs follow from its
    maps and bytes."""
    k = case["kind"]
    if k == "soft":
        return _exact_soft(case, seed)
    if k not in ("sgm", "dp", "agg"):
        return None
    W, H, D = case["W"], case["H"], case["D"]
    left, right, _ = _unit_pair(W, H, D, seed)
    if k == "sgm":
        return {"disp": None, "disp_norm": None,
                "dsi": _dsi64(left, right, D, "bt", 0).permute(1, 0, 2).contiguous()}
    if k == "dp":
        return {"disp": None, "disp_norm": None, "dsi": _dsi64(left, right, D, case["cost"], case["radius"])}
    # the aggregation of the float DSI that the call is given
    C = api.default_context().cost(left, right, D, kind=case["cost"], radius=case["radius"])
    C = C.double().view(H * W, D)
    S = torch.zeros_like(C)
    for dx, dy in _DIRS[:case["paths"]]:
        S += _walk64(C, float(np.float32(0.05)), float(np.float32(0.7)), dx, dy, W, H)
    return {"disp": None, "S": S.view(H, W, D), "subpixel": None}
