"""The rule that gives a tile several threads per pixel (vis.cu: vis_groups), at the
exact counts of whole tiles where it changes on this GPU: the last frame with twice
the threads and the first one without, whose buffers equal the counting variant's
(always one thread per pixel)."""
from __future__ import annotations

import re
from pathlib import Path

import numpy as np
import pytest

import tg_gb300 as tg
from scenes import fuzz_scene

pytestmark = pytest.mark.gpu

SOURCE = (Path(__file__).resolve().parents[1] / "tg_gb300" / "csrc" / "vis.cu").read_text()
TWO, MORE = (int(x) for x in re.search(r"<= \(g == 1u \? (\d+)u : (\d+)u\) \* unit", SOURCE).groups())


def groups(pixels: int, n_tiles: int, sms: int) -> int:
    g = 1
    while g < 8 and pixels * g * 2 <= 1024 and n_tiles * pixels * g * 2 <= (TWO if g == 1 else MORE) * 1024 * sms:
        g *= 2
    return g


@pytest.mark.parametrize("tile,step", [(t, g) for t in ((8, 8), (16, 8), (16, 16), (32, 16)) for g in (1, 2, 4)
                                       if t[0] * t[1] * g * 2 <= 1024])
def test_both_sides_of_a_step(tile, step):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pixels, rows = tile[0] * tile[1], 24
    cols = (TWO if step == 1 else MORE) * 1024 * sms // (pixels * 2 * step) // rows
    assert groups(pixels, rows * cols, sms) >= 2 * step and groups(pixels, rows * (cols + 1), sms) == step
    s = fuzz_scene(24, n_objects=12, box=30.0, max_cpa=4)
    with tg.Context(0, tile=tile) as ctx:
        sc = ctx.upload(s)
        for c in (cols, cols + 1):
            w, h = c * tile[0], rows * tile[1]
            view = tg.make_view((0.0, 5.0, -40.0), 0.1, float(np.pi), 0.9, w, h, 0.1, 300.0)
            out = torch.empty((2, w * h), dtype=torch.int64, device="cuda").fill_(7)
            torch.cuda.synchronize()
            for count in (0, 1):
                ctx.vis_count_work(bool(count))
                ctx.vis_render(sc, view, [out[count]])
            ctx.sync()
            assert torch.equal(out[0], out[1])
            assert (out[0] != -1).sum() > w * h // 50
        assert ctx.device_error().code == 0
        sc.close()
