"""Clusters that cover many tiles (vis.cu: the chunk list of the counting and
binning passes): cameras in and next to clusters, rectangles on both sides of 64
tiles and of the 256 tiles of a chunk, and more chunks than the list holds.  The
buffer equals the one of the record scan, which uses no bins; small frames also
equal the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import tg_gb300 as tg
from oracle_lib import Oracle
from scenes import fuzz_scene

pytestmark = pytest.mark.gpu


def render(s, view, n, tile, flags=0):
    import torch
    with tg.Context(0, tile=tile, flags=flags) as ctx:
        sc = ctx.upload(s)
        out = torch.full((n,), 7, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        for _ in range(2):                        # sized exactly, then from the frame before
            ctx.vis_render(sc, view, [out])
        ctx.sync()
        assert ctx.device_error().code == 0
        entries = ctx.vis_stats().bin_entries
        sc.close()
    return out.cpu().numpy().view(np.uint64), entries


@pytest.mark.parametrize("w,h", [(64, 64), (72, 64), (128, 128), (136, 128), (200, 150), (256, 256), (640, 360)])
@pytest.mark.parametrize("pos", [(0.0, 5.0, -20.0), (1.7, 2.3, -3.1)])
def test_near_clusters_over_many_tiles(w, h, pos):
    s = fuzz_scene(41, n_objects=8, box=12.0, max_cpa=3)
    view = tg.make_view(pos, 0.1, float(np.pi), 1.1, w, h, 0.1, 300.0)
    got, entries = render(s, view, w * h, (8, 8))
    assert entries > 0
    assert np.array_equal(got, render(s, view, w * h, (8, 8), tg.FLAG_MIN_BIN_CAPACITY)[0])
    if w * h <= 128 * 128:
        assert np.array_equal(got, Oracle().vis_render(s, view, mode=1))


def test_more_chunks_than_the_list_holds():
    # the clusters around the camera's plane cover all 32,400 tiles, 127 chunks each; the list holds 65,536
    s = tg.generate_scene(0, 1, 32, 32, seed=5, bernoulli_p=0.02, translation=(0.0, 0.0, 0.0))
    view = tg.make_view((0.3, 0.2, 0.1), 0.2, 0.7, 3.0, 1920, 1080, 0.1, 300.0)
    got, entries = render(s, view, 1920 * 1080, (8, 8))
    assert entries > 65536 * 256
    assert np.array_equal(got, render(s, view, 1920 * 1080, (8, 8), tg.FLAG_MIN_BIN_CAPACITY)[0])
