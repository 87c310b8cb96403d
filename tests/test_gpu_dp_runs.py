"""The DP scanline with whole vectors per lane (D a multiple of 16) and beside
it, around the load ring and the backtrack's stages, against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["hwd", "ref"])
@pytest.mark.parametrize("W,H,D", [(1, 5, 16), (2, 3, 32), (17, 4, 48), (31, 5, 64), (32, 4, 64), (33, 6, 64),
                                   (65, 3, 80), (96, 5, 128), (97, 2, 144), (130, 3, 256), (40, 4, 72), (64, 1, 16)])
def test_dp_runs(ctx, orc, layout, W, H, D):
    rng = np.random.default_rng(W + H + D)
    C = rng.integers(0, 6, size=(H, W, D)).astype(np.float32) / 2  # many ties
    C[rng.random(C.shape) < 0.05] = np.inf
    C[rng.random(C.shape) < 0.003] = np.nan
    lay = orc.LAYOUT_HWD if layout == "hwd" else orc.LAYOUT_REF_WHD
    V = C if layout == "hwd" else np.ascontiguousarray(C.transpose(1, 0, 2))
    want = orc.dp(V, lay)
    want = want[0] if isinstance(want, tuple) else want
    for offset in (0, 1):  # on and off 16 bytes
        buf = torch.empty(V.size + offset, device="cuda")
        t = buf[offset:].view(V.shape)
        t.copy_(torch.from_numpy(V))
        np.testing.assert_array_equal(ctx.dp(t, layout=layout)["disp"].cpu().numpy(), want)
