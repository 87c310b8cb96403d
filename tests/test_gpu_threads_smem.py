"""Host threads with contexts of their own and images of different widths: the
kernels' shared-memory limit is an attribute of the process, and a call never
finds it below what it needs."""
import threading

import numpy as np
import pytest
import torch

from thundervision_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["fused", "batch120", "batch300"])
def test_widths_side_by_side(kind):
    rng = np.random.default_rng(0)
    errors, go = [], threading.Barrier(2)

    def work(W, n):
        try:
            torch.cuda.set_device(0)
            ctx = api.Context(0)
            l, r = [torch.from_numpy(rng.integers(0, 256, size=(2, W)).astype(np.uint8)).cuda() for _ in range(2)]
            with torch.cuda.stream(torch.cuda.Stream()):
                b = None if kind == "fused" else api.Batch(ctx, [(l, r, 16, 1)], 10, int(kind[5:]))
                call = (lambda: ctx.stereo_sgm(l, r, 16, 10, 120, lr=1)) if b is None else b.run
                call()
                torch.cuda.current_stream().synchronize()
                go.wait()
                for _ in range(n):
                    call()
                torch.cuda.current_stream().synchronize()
            if b is not None:
                b.close()
            ctx.close()
        except Exception as e:  # handed to the test's thread
            errors.append(e)
            go.abort()

    threads = [threading.Thread(target=work, args=(W, 150)) for W in (16384, 8256)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert errors == []
