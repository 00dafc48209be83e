"""Entries dropped for a whole warp of pixels (vis.cu: warp_rays, warp_may_hit)
and the pair evaluation behind them.

On the CPU: the rule, restated in float32, never drops a cube that the exact
box test (ray_aabb, visibility.frag:22-52) finds on one of the warp's rays, for
rotations and other linear maps, near, touching and far origins, narrow and wide
bundles, and directions with zero components.  On the GPU: frames whose warps are narrow, wide,
cut off by the view's edge or axis-aligned, and cameras in and on cubes, equal the
oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import tg_gb300 as tg
from oracle_lib import Oracle
from scenes import fuzz_scene

f32 = np.float32


def may_hit(L, d, o):
    """warp_may_hit for the warp of rays d (32, 3), per entry (L (n, 3, 3), o (n, 3))."""
    lo, hi = d.min(0), d.max(0)
    m = f32(0.5) * (lo + hi)
    h = f32(0.5) * (hi - lo) * f32(1.00001) + f32(2e-6) * np.abs(m)
    u = (L[..., 0] * m[0] + (L[..., 1] * m[1] + L[..., 2] * m[2])).astype(f32)
    s = (np.abs(L[..., 0]) * h[0] + (np.abs(L[..., 1]) * h[1] + np.abs(L[..., 2]) * h[2])).astype(f32)
    c = f32(4.0) - o
    a = f32(1e-5) * np.abs(c) + f32(4.001)
    miss = np.zeros(len(o), bool)
    for j in range(3):
        k = (j + 1) % 3
        r = s[:, j] * (np.abs(c[:, k]) + a[:, k]) + s[:, k] * (np.abs(c[:, j]) + a[:, j]) + np.abs(u[:, j]) * a[:, k] + np.abs(u[:, k]) * a[:, j]
        miss |= np.abs(u[:, j] * c[:, k] - u[:, k] * c[:, j]) > r
    low = np.abs(u).max(1)
    return ~miss | ~((low > f32(1e-15)) & (low + s.max(1) < f32(1e15)))


def box_test(L, d, o):
    """The exact test of every (entry, ray) pair: the shader's direction and ray_aabb, float32."""
    with np.errstate(all="ignore"):
        u = [((L[:, None, i, 0] * d[None, :, 0] + L[:, None, i, 1] * d[None, :, 1]) + L[:, None, i, 2] * d[None, :, 2]).astype(f32)
             for i in range(3)]
        mag = np.sqrt((u[0] * u[0] + u[1] * u[1]) + u[2] * u[2])
        near, far = np.full(mag.shape, -np.inf, f32), np.full(mag.shape, np.inf, f32)
        beside = np.zeros(mag.shape, bool)
        for i in range(3):
            di, oi = u[i] / mag, o[:, None, i] + np.zeros_like(mag)
            zero = di == 0
            t0, t1 = (f32(0.0) - oi) / di, (f32(8.0) - oi) / di
            near = np.where(zero, near, np.maximum(near, np.minimum(t0, t1)))
            far = np.where(zero, far, np.minimum(far, np.maximum(t0, t1)))
            beside |= zero & ((oi < 0) | (oi > 8))
        return (far > 0) & (near <= far) & ~beside


@pytest.mark.parametrize("spread", [0.0, 1e-5, 1e-3, 0.03, 0.4, 3.0])
@pytest.mark.parametrize("linear", ["rotation", "identity", "any", "tiny", "huge"])
def test_no_entry_is_dropped_that_a_ray_meets(spread, linear):
    rng = np.random.default_rng([int(spread * 1e6), len(linear)])
    n = 3000
    hits = 0
    for _ in range(12):
        M = rng.normal(size=(n, 3, 3))
        if linear == "rotation":
            M = np.linalg.qr(M)[0]
        elif linear == "identity":
            M = np.broadcast_to(np.eye(3), (n, 3, 3))
        elif linear != "any":
            M = M * 10.0 ** rng.uniform(*((-25, -5) if linear == "tiny" else (5, 25)), (n, 1, 1))
        L = M.astype(f32)
        mid = rng.normal(size=3)
        mid /= np.linalg.norm(mid)
        if linear == "identity":
            mid = np.eye(3)[rng.integers(3)]
        d = (mid + spread * rng.uniform(-0.5, 0.5, (32, 3))).astype(f32)
        if linear == "identity":
            d[:16, rng.integers(3)] = 0.0
        # origins such that points on and around the cube's surface lie along some ray
        ray = np.einsum("nij,nj->ni", M, d[rng.integers(32, size=n)].astype(np.float64))
        ray /= np.maximum(np.linalg.norm(ray, axis=1, keepdims=True), 1e-300)
        at = rng.uniform(-0.2, 8.2, (n, 3))
        face = rng.integers(3, size=n)
        at[np.arange(n), face] = rng.choice([0.0, 8.0], n)
        at = np.where(rng.uniform(size=(n, 1)) < 0.5, at, np.round(at))
        away = rng.uniform(-40, 40, (n, 3)) * (rng.uniform(size=(n, 1)) < 0.3)
        o = (at + away - ray * np.where(rng.uniform(size=(n, 1)) < 0.2, 0.0, 10.0 ** rng.uniform(-3, 5, (n, 1)))).astype(f32)
        with np.errstate(all="ignore"):
            keep = may_hit(L, d, o)
        hit = box_test(L, d, o).any(1)
        assert not (hit & ~keep).any()
        hits += hit.sum()
    assert hits > 1000 or linear in ("tiny", "huge")


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(1, 1), (7, 5), (33, 9), (64, 65), (131, 3)])
@pytest.mark.parametrize("fov", [0.02, 1.1, 3.0])
@pytest.mark.parametrize("where", ["outside", "in a cube", "on a face"])
def test_frames_equal_the_oracle(size, fov, where):
    import torch
    scenes = [fuzz_scene(31, n_objects=5, box=25.0, max_cpa=3),
              tg.generate_scene(0, 1, 4, 4, seed=3, bernoulli_p=0.2, translation=(0.0, 0.0, 0.0))]
    pos, yaw = {"outside": ((0.0, 1.0, -60.0), float(np.pi)), "in a cube": ((1.7, 2.3, -3.1), 2.0), "on a face": ((0.0, 8.0, -8.0), 0.0)}[where]
    w, h = size
    view = tg.make_view(pos, 0.0 if where == "on a face" else 0.1, yaw, fov, w, h, 0.1, 300.0)
    for s in scenes:
        want = Oracle().vis_render(s, view, mode=1)
        for tile in ((8, 8), (16, 16), (32, 1)):
            with tg.Context(0, tile=tile) as ctx:
                sc = ctx.upload(s)
                out = torch.empty(w * h, dtype=torch.int64, device="cuda")
                for count in (True, False):
                    out.fill_(7)
                    torch.cuda.synchronize()
                    ctx.vis_count_work(count)
                    ctx.vis_render(sc, view, [out])
                    ctx.sync()
                    assert np.array_equal(out.cpu().numpy().view(np.uint64), want)
                assert ctx.device_error().code == 0
                sc.close()
