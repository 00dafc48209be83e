"""The SVO build's rules against the oracle, voxels and materials bit for bit:
many objects of different LUTs over the same blocks (the order of a block's
pairs decides its materials), matrices with and without a usable inverse, an
unrotated object on whole coordinates, blocks whose side is and is not exactly 32
(the layer split), and updates, which split every block, against the oracle's
build of the moved scene.  And the memory pool behind the arrays: rebuilt arrays
hold nothing of the last SVO, threads with a context each, memory given back."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import tg_gb300 as tg
from oracle_lib import Oracle, OracleSvo, gi_render, svo_build_with_materials
from scenes import fuzz_scene

pytestmark = pytest.mark.gpu


def make(kind, seed, centre, spread, n=10, n_luts=4):
    s = fuzz_scene(seed, n_objects=n, box=spread, max_cpa=3, density=0.4)
    rng = np.random.default_rng(seed)
    o = s.objects.copy()
    o["translation"] += np.asarray(centre, np.float32)
    R = o["rotation"].reshape(n, 4, 4)
    if kind == "odd":
        R[0] *= 0.7                            # (the candidate pass takes no cluster for larger than 8 voxels a side)
        R[1][:3, :3] *= 0.3
        R[2][0] = R[2][1]                      # singular
        R[3] *= 1e8
        R[4][:3, :3] += rng.normal(scale=0.3, size=(3, 3))
        R[5] = np.eye(4)
        o["translation"][5] = np.round(o["translation"][5])
    elif kind == "unrotated":
        R[:] = np.eye(4)
        o["translation"] = np.round(o["translation"])
    o["rotation"] = R.reshape(n, 16)
    o["lut_idx"] = np.arange(n) % n_luts
    luts = np.concatenate([s.luts[:256]] * n_luts)
    for k in range(n_luts):
        luts["albedo"][256 * k:256 * (k + 1)] *= np.float32(1.0 - 0.2 * k)
    return tg.HostScene(o, s.cluster_pointers, s.cluster_idx_to_object_idx, s.voxel_bits, s.material_idx, luts)


def assert_oracle(ctx, s, sc, svo, mn, L, centre):
    import torch
    ora = Oracle()
    xyz, words, mats = svo_build_with_materials(ora, s, mn, L, capacity=1 << 12)
    got_xyz, got_words = svo.download()
    assert len(xyz) > 0
    assert np.array_equal(got_xyz, xyz) and np.array_equal(got_words, words)
    # materials through path tracing from random visibility words
    w, h = 64, 48
    view = tg.make_view((centre[0], centre[1], centre[2] - 1.2 * 2 ** (L - 1)), 0.0, float(np.pi), 1.2, w, h, 0.1, 4.0 * 2 ** L)
    rng = np.random.default_rng(1)
    vis = ((rng.integers(0, 1 << 23, w * h).astype(np.uint64) << np.uint64(40)) |
           (rng.integers(0, len(s.cluster_pointers), w * h).astype(np.uint64) << np.uint64(9)) |
           rng.integers(0, 512, w * h).astype(np.uint64))
    par = tg.gi_params(spp=2, bounces=2, seed=3, max_steps=256)
    rgb = torch.empty(w * h * 3, dtype=torch.float32, device="cuda")
    ctx.gi_render(sc, svo, view, torch.from_numpy(vis.view(np.int64)).cuda(), par, rgb)
    ctx.sync()
    assert ctx.device_error().code == 0
    osvo = OracleSvo(ora, xyz, words, mats, np.asarray(mn, np.float32), L)
    want = gi_render(ora, osvo, s, view, par, vis)
    osvo.close()
    assert np.array_equal(rgb.cpu().numpy().reshape(-1, 3).view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("kind", ["rotated", "odd", "unrotated"])
@pytest.mark.parametrize("L,centre,spread", [
    (8, (0, 0, 0), 15.0), (9, (0, 0, 0), 120.0), (6, (0, 0, 0), 20.0),
    (7, (16777216 - 128, 1000, -16777216 + 64), 30.0),      # every side 32, at the last whole coordinates
    (7, (16777216 - 32, 1000, 0), 20.0),                    # sides beyond 2^24
])
def test_build_and_updates_equal_the_oracle(kind, L, centre, spread):
    mn = [float(min(max(c - 2 ** (L - 1), -16777216), 16777216)) for c in centre]
    s = make(kind, L, centre, spread)
    rng = np.random.default_rng(L)
    with tg.Context(0) as ctx:
        sc = ctx.upload(s)
        svo = ctx.svo_build(sc, mn, L)
        assert_oracle(ctx, s, sc, svo, mn, L, centre)
        for idx in ([1], [0, 4, 5]):
            o = s.objects.copy()
            o["translation"][idx] += np.round(rng.uniform(-spread / 2, spread / 2, (len(idx), 3))).astype(np.float32)
            s = tg.HostScene(o, s.cluster_pointers, s.cluster_idx_to_object_idx, s.voxel_bits, s.material_idx, s.luts)
            sc.set_objects(0, o)
            assert svo.update(sc) >= 1
            assert_oracle(ctx, s, sc, svo, mn, L, centre)
        svo.close()
        sc.close()


def test_arrays_of_a_closed_svo_are_reused_without_a_trace():
    with tg.Context(0) as ctx:
        for seed, L in ((1, 9), (2, 8), (3, 9), (1, 9)):
            s = make("rotated", seed, (0, 0, 0), 60.0)
            mn = [-(2.0 ** (L - 1))] * 3
            sc = ctx.upload(s)
            svo = ctx.svo_build(sc, mn, L)
            assert_oracle(ctx, s, sc, svo, mn, L, (0, 0, 0))
            svo.close()
            sc.close()


def test_threads_build_and_free_side_by_side():
    s = make("rotated", 7, (0, 0, 0), 80.0)
    mn = [-256.0] * 3
    xyz, words, _ = svo_build_with_materials(Oracle(), s, mn, 9, capacity=1 << 12)
    failures = []

    def work():
        try:
            with tg.Context(0) as ctx:
                sc = ctx.upload(s)
                for _ in range(5):
                    svo = ctx.svo_build(sc, mn, 9)
                    got = svo.download()
                    svo.close()
                    assert np.array_equal(got[0], xyz) and np.array_equal(got[1], words)
                sc.close()
        except Exception as e:                  # noqa: BLE001 (reported by the main thread)
            failures.append(e)

    threads = [threading.Thread(target=work) for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def test_a_context_gives_its_pool_back():
    import torch
    s = make("rotated", 9, (0, 0, 0), 100.0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        with tg.Context(0) as ctx:
            sc = ctx.upload(s)
            svo = ctx.svo_build(sc, [-256.0] * 3, 9)
            assert svo.info().n_blocks > 0
            svo.close()
            sc.close()
        held = before - torch.cuda.mem_get_info()[0]
    # three contexts leave no more than one of them could have kept by the driver's own granularity
    assert held < 64 << 20
