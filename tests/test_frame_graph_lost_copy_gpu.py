"""A tile of a frame graph whose staging copy never lands (the host flag that makes
its first batch wait for bytes nobody copies): its CTA gives up after a second,
and by then holds the next item of the work queue.  That tile is still rendered:
only the timed-out tile of the first job's one-tile view is incomplete, all other
jobs' buffers are whole, and the status word says what happened."""
from __future__ import annotations

import numpy as np
import pytest

import tg_gb300 as tg

pytestmark = pytest.mark.gpu


def test_only_the_tile_whose_copy_is_lost_is_incomplete():
    import torch
    s = tg.generate_scene(0, 1, 12, 12, seed=5, bernoulli_p=0.2, translation=(0.0, 0.0, 0.0))
    view = lambda w, h: tg.make_view((0.3, 0.2, 0.1), 0.2, 0.7, 1.3, w, h, 0.1, 300.0)
    # 16x16 tiles: one, and more than the queue kernel's CTAs take in two rounds (5 on each SM)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    w, h = 1024, 16 * ((2 * 5 * sms) // 64 + 8)
    jobs = [view(16, 16), view(w, h)]
    outs = [torch.empty(n, dtype=torch.int64, device="cuda") for n in (256, w * h)]
    want = torch.empty_like(outs[1])
    with tg.Context(0) as ctx:
        sc = ctx.upload(s)
        ctx.vis_render(sc, jobs[1], [want])
        ctx.sync()
        sc.close()
    tiles = want.cpu().numpy().view(np.uint64).reshape(h // 16, 16, w // 16, 16)
    assert ((tiles != np.uint64(tg.VIS_EMPTY)).any(axis=(1, 3))).all()      # every tile has entries
    with tg.Context(0, flags=tg.FLAG_TEST_LOST_COPY) as ctx:
        sc = ctx.upload(s)
        g = ctx.frame_graph([(sc, v, [o]) for v, o in zip(jobs, outs)])     # sized by frames that lose copies
        ctx.sync()
        assert ctx.device_error().code == 5
        for o in outs:
            o.fill_(7)
        torch.cuda.synchronize()
        g.launch()
        ctx.sync()
        err = ctx.device_error()
        assert (err.code, err.where) == (5, 5)
        assert torch.equal(outs[1], want)
        assert (outs[0] != 7).all()
        g.close()
        sc.close()
