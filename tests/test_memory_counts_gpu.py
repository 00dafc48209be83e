"""The bytes that the library says it holds: every array of a scene store counts
against the context's budget, every per-slot array in an SVO's device_bytes."""
from __future__ import annotations

import pytest

import tg_gb300 as tg
from scenes import fuzz_scene

pytestmark = pytest.mark.gpu


def scene_bytes(s) -> int:
    n, p, c = len(s.objects), len(s.cluster_pointers), s.n_clusters
    # objects with the rotation's inverse (3x3, and whole); pointers with their table; clusters
    return n * (96 + 36 + 64) + p * (4 + 4) + c * (4 + 64 + 512) + len(s.luts) * 16


def test_every_scene_array_counts_against_the_budget():
    s = fuzz_scene(81, n_objects=40, box=60.0, max_cpa=2)
    with tg.Context(0) as c:
        sc = c.upload(s)
        assert c.memory()[1] == scene_bytes(s)
        sc.close()
        c.set_memory_budget(scene_bytes(s) - 1)
        with pytest.raises(tg.TgxError) as e:
            c.upload(s)
        assert e.value.status == 2 and c.memory()[1] == 0
        c.set_memory_budget(scene_bytes(s))
        sc = c.upload(s)
        sc.set_objects(0, s.objects)
        assert c.memory()[1] == scene_bytes(s)
        sc.close()
        assert c.memory()[1] == 0


@pytest.mark.parametrize("materials", [True, False])
def test_svo_bytes_are_its_arrays(ctx, materials):
    s = fuzz_scene(82, n_objects=6, box=60.0, max_cpa=4)
    L = 8
    sc = ctx.upload(s)
    svo = ctx.svo_build(sc, [-128.0] * 3, L, materials=materials)
    i = svo.info()
    table = i.blocks_per_axis ** 3
    pyramid = sum(((i.blocks_per_axis >> k) ** 3 + 31) // 32 for k in range(L - 4))
    # voxels, sub-block masks, non-empty flag, free list, block, codes
    slot = 4096 + 128 + 4 + 4 + 4 + (65536 if materials else 0)
    assert i.device_bytes == 4 * table + i.n_blocks * slot + 4 * pyramid + 96 * len(s.objects)
    svo.close()
    sc.close()
