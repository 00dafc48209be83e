"""Closing an SVO waits for every stream of the device: another context may still
traverse it, and its arrays go back to a pool that the next build takes them
from.  A long batch of traces is queued on one context, another one closes the SVO
(or nobody's context does) and builds the next; the close returns only after the
traces, and these found what they find when they run alone."""
from __future__ import annotations

import numpy as np
import pytest

import tg_gb300 as tg
from scenes import fuzz_scene

pytestmark = pytest.mark.gpu

MN, L, RAYS = [-256.0] * 3, 9, 500_000


@pytest.mark.parametrize("closer", ["the building context", "no context"])
def test_close_waits_for_another_contexts_traces(closer):
    import torch
    rng = np.random.default_rng(4)
    o = torch.tensor(rng.uniform(-200, 200, (RAYS, 3)).astype(np.float32), device="cuda")
    d = rng.normal(size=(RAYS, 3))
    d = torch.tensor((d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32), device="cuda")
    alone, queued = [(torch.empty(RAYS, dtype=torch.float32, device="cuda"),
                      torch.empty((RAYS, 3), dtype=torch.int32, device="cuda")) for _ in range(2)]
    with tg.Context(0) as a, tg.Context(0) as b:
        scenes = [a.upload(fuzz_scene(k, n_objects=40, box=150.0, max_cpa=6)) for k in (51, 52)]
        svo = a.svo_build(scenes[0], MN, L)
        a.sync()
        seen_by_b = tg.Svo(b, svo.handle)
        torch.cuda.synchronize()
        seen_by_b.trace(o, d, *alone, max_steps=512)
        b.sync()
        assert (alone[0] < 1e30).sum() > RAYS // 100
        done = torch.cuda.Event()
        for _ in range(600):
            seen_by_b.trace(o, d, *queued, max_steps=512)
        done.record(torch.cuda.ExternalStream(b.stream))
        assert not done.query()                     # else the close has nothing to wait for
        seen_by_b.handle = None
        tg.lib.tgx_svo_destroy(a.handle if closer == "the building context" else None, svo.handle)
        svo.handle = None
        assert done.query()
        following = a.svo_build(scenes[1], MN, L)
        a.sync()
        b.sync()
        for x, y in zip(alone, queued):
            assert torch.equal(x, y)
        assert a.device_error().code == 0 and b.device_error().code == 0
        following.close()
        for sc in scenes:
            sc.close()
