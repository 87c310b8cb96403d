"""The accumulating kernels, which run where penalties exceed 127.5 (and where
the scratch of the directions stored apart is refused): the batch's tile
variants, queue, trace, autotuner and error paths, and the single pair's passes
at edge sizes, under every recurrence and at larger frames, against per-pair
calls and the oracle (bit-exact)."""
import numpy as np
import pytest
import torch

import test_gpu_batch as batches
import test_gpu_dirs as pairs_
from thundervision_b200 import Batch

pytestmark = pytest.mark.gpu

P2 = 128


@pytest.fixture()
def wide_penalty(monkeypatch):
    """The batch tests' helpers with a penalty that accumulates."""
    def per_pair(ctx, pairs, paths=8):
        return [ctx.stereo_sgm(l, r, D, 10, P2, paths=paths, lr=lr, norm=True, right_disp=lr is not None)
                for (l, r, D, lr) in pairs]

    monkeypatch.setattr(batches, "_per_pair", per_pair)
    monkeypatch.setattr(batches, "_batch", lambda ctx, pairs, paths=8: Batch(ctx, pairs, 10, P2, paths=paths, norm=True,
                                                                             right_disp="lr"))


TILES = [{}, {"lines_per_cta": 3, "rows_per_cta": 1, "order": 1}, {"split_disparity": 1, "rows_per_cta": 5},
         {"lines_per_cta": 24, "rows_per_cta": 25, "split_disparity": 1},
         {"lines_per_cta": 7, "rows_per_cta": 12, "split_disparity": 0}, {"ctas_per_sm": 2},
         {"ctas_per_sm": 2, "lines_per_cta": 24, "rows_per_cta": 25, "split_disparity": 1}]


@pytest.mark.parametrize("paths", [8, 4])
@pytest.mark.parametrize("tiles", TILES)
def test_batch_tiles(ctx, wide_penalty, paths, tiles):
    batches.test_batch_matches_per_pair(ctx, paths, tiles)


@pytest.mark.parametrize("name", ["trace", "graph_replay_video", "autotune_keeps_results", "queue_layout",
                                  "bad_work_item_is_rejected", "unsatisfied_dependency_times_out"])
def test_batch_runtime(ctx, wide_penalty, name):
    getattr(batches, "test_batch_" + name)(ctx)


SEMS = [("standard", "full"), ("ref_cpu", "ref"), ("ref_gpu", "ref")]


@pytest.mark.parametrize("sem,table", SEMS)
@pytest.mark.parametrize("W,H,D,paths,lr", [
    (47, 33, 16, 8, 1), (49, 48, 17, 4, 1), (24, 70, 32, 8, None), (97, 5, 33, 8, 0), (64, 64, 64, 8, 1),
    (129, 31, 65, 4, None), (70, 41, 128, 8, 1), (33, 90, 129, 8, 1), (261, 18, 256, 8, 1), (300, 37, 200, 4, 2),
    (12, 300, 8, 8, 1), (1, 40, 16, 8, 1), (40, 1, 40, 8, 1), (3, 2, 2, 8, 1), (31, 29, 250, 8, None),
    (640, 480, 64, 8, 1),
])
def test_edges(ctx, orc, sem, table, W, H, D, paths, lr):
    pairs_._check(ctx, orc, W, H, D, p2=200, paths=paths, sem=sem, table=table, lr=lr, seed=(W + H) % 2)


@pytest.mark.parametrize("sem,table", SEMS[:2])
def test_full_hd(ctx, orc, sem, table):
    pairs_._check(ctx, orc, 1920, 270, 256, p2=200, sem=sem, table=table)


def test_path_taken(ctx):
    l = torch.zeros((40, 60), dtype=torch.uint8, device="cuda")
    for p2, apart in ((127.5, True), (128, False)):
        names = [n for n, _ in ctx.kernel_times(lambda: ctx.stereo_sgm(l, l, 16, 10, p2, lr=1))]
        assert ("fused_sum_wta" in names) == apart
