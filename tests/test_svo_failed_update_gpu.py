"""An update that fails once its blocks have slots (on the host: a flag of the
context that runs it) leaves an SVO that can be used: no block but those of before,
with their voxels, and a pyramid that fits them (by the oracle's traversal of the
downloaded blocks), also after updates that succeed."""
from __future__ import annotations

import numpy as np
import pytest

import tg_gb300 as tg
from oracle_lib import Oracle, OracleSvo
from scenes import fuzz_scene

pytestmark = pytest.mark.gpu

MN, L = [-256.0] * 3, 9


def blocks(svo):
    xyz, words = svo.download()
    return {tuple(p): w for p, w in zip(xyz.tolist(), words)}


def assert_consistent(ctx, svo):
    """The SVO's counts and a batch of traces are those of the blocks it downloads."""
    import torch
    n = 20000
    rng = np.random.default_rng(8)
    o = rng.uniform(-250, 250, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    t = torch.empty(n, dtype=torch.float32, device="cuda")
    v = torch.empty((n, 3), dtype=torch.int32, device="cuda")
    do, dd = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    torch.cuda.synchronize()
    svo.trace(do, dd, t, v, max_steps=4096)
    ctx.sync()
    assert ctx.device_error().code == 0
    xyz, words = svo.download()
    assert svo.info().n_nonempty_blocks == len(xyz) > 0
    osvo = OracleSvo(Oracle(), xyz, words, None, np.asarray(MN, np.float32), L)
    want_t, want_v = osvo.trace(o, d, 4096)[:2]
    osvo.close()
    assert np.array_equal(t.cpu().numpy(), want_t) and np.array_equal(v.cpu().numpy(), want_v)
    assert (want_t < 1e30).sum() > 50


@pytest.mark.parametrize("materials", [True, False])
@pytest.mark.parametrize("far", [20.0, 200.0])          # blocks of before, and many new ones (the arrays grow)
def test_a_failed_update_leaves_the_rest(materials, far):
    s = fuzz_scene(71, n_objects=30, box=60.0, max_cpa=5)
    rng = np.random.default_rng(2)
    with tg.Context(0) as ctx, tg.Context(0, flags=tg.FLAG_TEST_FAILED_FILL) as failing:
        sc = ctx.upload(s)
        with pytest.raises(tg.TgxError) as e:
            failing.svo_build(sc, MN, L, materials=materials)
        assert e.value.status == 3
        svo = ctx.svo_build(sc, MN, L, materials=materials)
        before = blocks(svo)
        o = s.objects.copy()
        o["translation"][:10] += rng.uniform(-far, far, (10, 3)).astype(np.float32)
        sc.set_objects(0, o)
        theirs = tg.Svo(failing, svo.handle)
        with pytest.raises(tg.TgxError) as e:
            theirs.update(sc)
        theirs.handle = None
        assert e.value.status == 3
        failing.sync()
        left = blocks(svo)
        assert 0 < len(left) < len(before)
        for p, w in left.items():
            assert np.array_equal(w, before[p])
        assert_consistent(ctx, svo)
        # another object: the update succeeds, over the blocks that are left
        o["translation"][20] += np.float32(31.0)
        sc.set_objects(0, o)
        assert svo.update(sc) == 1
        assert_consistent(ctx, svo)
        # and the objects of the failed one come back when they move again
        o["translation"][:10] = s.objects["translation"][:10]
        sc.set_objects(0, o)
        assert svo.update(sc) == 10
        fresh = ctx.svo_build(sc, MN, L, materials=materials)
        for x, y in zip(svo.download(), fresh.download()):
            assert np.array_equal(x, y)
        assert svo.info().n_blocks == fresh.info().n_blocks
        fresh.close()
        svo.close()
        sc.close()
