"""The traversal's fast form (svo_trace.cuh) against the oracle's form.

On the CPU: one point location at voxel resolution, mirrored and clamped to a
cell, gives the same child at every finer level as locating and clamping level
by level; and the level a step ascends to, from the trailing zeros of the new
coordinate, is the one the level-by-level climb finds.  On the GPU: ray batches
of every size class of the persistent kernel, and rays on both sides of the
rule that picks the fast form, equal the oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from test_trace_ascend import climb, level_log2, n_levels

f32 = np.float32
MAGIC = f32(12582912.0)


def round_down(x):
    """The largest float32 <= x (float64)."""
    y = x.astype(f32)
    return np.where(y.astype(np.float64) > x, np.nextafter(y, f32(-np.inf)), y).astype(f32)


def cell_at(p, g, step, lo, hi):
    x = p * f32(2.0 ** -g)
    f = np.floor(x)
    f = np.where((step < 0) & (x == f), f - f32(1.0), f)
    return np.clip(f.astype(np.int64), lo, hi)


@pytest.mark.parametrize("L", range(6, 15))
def test_one_location_serves_every_finer_level(L):
    rng = np.random.default_rng(L)
    E, NL, n = 1 << L, n_levels(L), 4000
    for top in range(NL):
        g = level_log2(L, top)
        c = rng.integers(0, E >> g, n)                    # the current cell, real coordinates
        p = ((c + rng.uniform(-0.1, 1.1, n)) * (1 << g)).astype(f32)
        p[::2] = np.round(p[::2])                         # points on cell borders
        p[1::8] = np.nextafter(p[1::8], f32(np.inf))
        p[3::8] = rng.uniform(-2.0 ** 20, 2.0 ** 20, p[3::8].shape).astype(f32)
        step = rng.choice([-1, 1], n)
        neg = step < 0
        pm = np.where(neg, -p, p)
        at = round_down(pm.astype(np.float64) + MAGIC.astype(np.float64) + np.where(neg, E, 0))
        at = (at.view(np.int32).astype(np.int64) - int(MAGIC.view(np.int32)))
        cm = np.where(neg, (E >> g) - 1 - c, c)           # the cell, mirrored
        v = np.clip(at, cm << g, ((cm + 1) << g) - 1)
        real = np.where(neg, E - 1 - v, v)
        for li in range(top - 1, -1, -1):                 # the oracle's descent, level by level
            gc, gp = level_log2(L, li), level_log2(L, li + 1)
            lo = c << (gp - gc)
            c = cell_at(p, gc, step, lo, lo + (1 << (gp - gc)) - 1)
            assert np.array_equal(real >> gc, c), (top, li)


def test_ascend_from_trailing_zeros_equals_the_climb():
    for L in range(6, 15):
        NL = n_levels(L)
        for li in range(NL):
            g = level_log2(L, li)
            for cur in range(1, 1 << (L - g)):            # mirrored: every step goes up
                w = cur << g
                p = (w & -w).bit_length() - 1
                up = 0
                while up < NL - 1 and level_log2(L, up + 1) < p + 1:
                    up += 1
                assert up == climb(L, NL, li, g, cur - 1, cur), (L, li, cur)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 128, 129, 4097, 136192, 136193, 300001])
def test_ray_batches_equal_the_oracle(n):
    """Sizes around a warp, a CTA, and the rays that the resident warps take by index before they use the queue."""
    import torch
    import tg_gb300 as tg
    from oracle_lib import Oracle, OracleSvo
    from scenes import fuzz_scene

    oracle = Oracle()
    s = fuzz_scene(5, n_objects=6, box=100.0, max_cpa=4)
    L, mn = 9, [-256.0] * 3
    blocks, words, _ = oracle.svo_build(s, mn, L)
    osvo = OracleSvo(oracle, blocks, words, None, mn, L)
    rng = np.random.default_rng(n)
    o = rng.uniform(-256.0, 256.0, (n, 3))
    d = rng.uniform(-90.0, 90.0, (n, 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o[::5] = np.round(o[::5])                             # lattice points
    d[::7, 0] = 0.0
    d[::11, 1:] = 0.0
    d[::13] *= 1e-19                                      # below the fast form's smallest component
    d[3::13] *= 1e-10                                     # above it
    d[5::13] *= 1e20
    far = np.arange(n) % 17 == 3                          # origins on both sides of 2^20 voxels
    o[far] -= d[far] / np.maximum(np.linalg.norm(d[far], axis=1, keepdims=True), 1e-30) * rng.choice(
        [5e4, 1.04e6, 1.06e6, 3e6], (int(far.sum()), 1))
    o, d = o.astype(f32), d.astype(f32)
    with tg.Context(0) as ctx:
        sc = ctx.upload(s)
        svo = ctx.svo_build(sc, mn, L)
        to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
        for steps in (0, 3, 7, 40, 4096):
            t = torch.empty(n, dtype=torch.float32, device="cuda")
            v = torch.empty((n, 3), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            svo.trace(to, td, t, v, max_steps=steps)
            ctx.sync()
            ot, ov, _, _ = osvo.trace(o, d, steps)
            assert np.array_equal(t.cpu().numpy().view(np.uint32), ot.view(np.uint32)), steps
            hit = ot < 3e38
            assert np.array_equal(v.cpu().numpy()[hit], ov[hit]), steps
        assert n < 100 or hit.sum() > n // 50
        svo.close()
        sc.close()
