"""What a context keeps of closed SVOs goes back to the device: when the program
asks (tgx_trim), and when an allocation of any context finds no room.  (The
failing one here asks for more than any device has, so nothing is filled up.)"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import tg_gb300 as tg
from scenes import fuzz_scene

pytestmark = pytest.mark.gpu


def free_bytes() -> int:
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture
def closed_svo():
    """A context that has closed an SVO of more than 128 MiB, and how much the device lost by that."""
    with tg.Context(0) as ctx:
        sc = ctx.upload(fuzz_scene(61, n_objects=400, box=230.0, max_cpa=8))
        ctx.svo_build(sc, [-256.0] * 3, 9).close()      # the scratch of a build is there from here on
        ctx.trim()
        before = free_bytes()
        svo = ctx.svo_build(sc, [-256.0] * 3, 9)
        assert svo.info().device_bytes > 128 << 20
        words = svo.download()
        svo.close()
        assert before - free_bytes() > 128 << 20
        yield ctx, sc, before, words
        sc.close()


def test_trim_gives_the_memory_back(closed_svo):
    ctx, sc, before, words = closed_svo
    ctx.trim()
    assert before - free_bytes() < 8 << 20
    svo = ctx.svo_build(sc, [-256.0] * 3, 9)            # and the next build is as good
    got = svo.download()
    assert np.array_equal(got[0], words[0]) and np.array_equal(got[1], words[1])
    ctx.trim()                                          # an update without the scratch of a build
    objects = fuzz_scene(61, n_objects=400, box=230.0, max_cpa=8).objects.copy()
    objects["translation"][:40] += np.float32(13.0)
    sc.set_objects(0, objects)
    assert svo.update(sc) == 40
    again = ctx.svo_build(sc, [-256.0] * 3, 9)
    for x, y in zip(svo.download(), again.download()):
        assert np.array_equal(x, y)
    assert ctx.device_error().code == 0
    svo.close()
    again.close()


@pytest.mark.parametrize("same_context", [True, False])
def test_an_allocation_without_room_gives_the_memory_back(closed_svo, same_context):
    ctx, sc, before, _ = closed_svo
    other = ctx if same_context else tg.Context(0)
    mine = sc if same_context else other.upload(fuzz_scene(62, n_objects=2, box=5.0, max_cpa=2))
    n = 16                                              # frames of 34 GB each in unpinned host memory
    views = np.concatenate([tg.make_view((0.0, 0.0, -40.0), 0.0, float(np.pi), 1.0, 65520, 65520, 0.1, 100.0)] * n)
    word = np.zeros(1, np.uint64)                       # never written: the call fails before
    outs = (C.c_void_p * n)(*[word.ctypes.data] * n)
    assert tg.lib.tgx_vis_render_host(other.handle, mine.handle, views.ctypes.data, n, outs) == 2
    scratch = 0 if same_context else 64 << 20
    assert before - free_bytes() < (64 << 20) + scratch
    small = np.zeros(64 * 64, np.uint64)
    other.vis_render_host(mine, tg.make_view((0.0, 0.0, -40.0), 0.0, float(np.pi), 1.0, 64, 64, 0.1, 100.0), [small])
    assert (small != 0).all()                           # the context goes on
    if not same_context:
        mine.close()
        other.close()
