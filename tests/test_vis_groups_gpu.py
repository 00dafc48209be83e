"""Frames on both sides of every step of the rule that gives a tile several
threads per pixel: the buffer equals the counting variant's (always one thread
per pixel), with normal bins, with bins that overflow into the record scan, and
written to pinned host memory; small frames also equal the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import tg_gb300 as tg
from oracle_lib import Oracle
from scenes import fuzz_scene

pytestmark = pytest.mark.gpu

# 12 * 1024 threads per SM over the tile's pixels and 2 threads each, 8 * 1024 with 4 or 8, on 152 SMs
EDGES = [m * 1024 * 152 // (2 * g) for m, g in ((12, 1), (8, 2), (8, 4))]


@pytest.mark.parametrize("tile", [(8, 8), (16, 8), (16, 16), (32, 16), (8, 4), (8, 12)])
@pytest.mark.parametrize("pixels", [37 * 29, *EDGES, *[e + 4096 for e in EDGES]])
def test_threads_per_pixel_change_no_word(tile, pixels):
    import torch
    s = fuzz_scene(23, n_objects=6, box=30.0, max_cpa=4)
    h = max(1, int((pixels * 0.6) ** 0.5) // tile[1] * tile[1])
    w = max(1, pixels // h)
    view = tg.make_view((0.0, 5.0, -70.0), 0.1, float(np.pi), 1.1, w, h, 0.1, 300.0)
    frames = []
    for flags in (0, tg.FLAG_MIN_BIN_CAPACITY):
        with tg.Context(0, tile=tile, flags=flags) as ctx:
            sc = ctx.upload(s)
            out = torch.empty(w * h, dtype=torch.int64, device="cuda")
            for count in (True, False):
                out.fill_(7)
                torch.cuda.synchronize()
                ctx.vis_count_work(count)
                ctx.vis_render(sc, view, [out])
                ctx.sync()
                frames.append(out.cpu().numpy().view(np.uint64).copy())
            host = torch.empty(w * h, dtype=torch.int64, pin_memory=True).numpy().view(np.uint64)
            ctx.vis_render_host(sc, view, [host])
            frames.append(host.copy())
            assert ctx.device_error().code == 0
            sc.close()
    for f in frames[1:]:
        assert np.array_equal(f, frames[0])
    assert (frames[0] != np.uint64(tg.VIS_EMPTY)).sum() > pixels // 50
    if pixels < 2000:
        assert np.array_equal(frames[0], Oracle().vis_render(s, view, mode=1))
