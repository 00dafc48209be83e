"""The primary surface of objects with every kind of matrix: the products the
decode leaves out (0 and 1 times the inverse) change nothing for rotated,
scaled, sheared, mirrored and projective matrices, and the ones whose inverse
is no moderate number take the full products.  Shading equals the oracle bit
for bit, over words of the frame and arbitrary words of every object."""
from __future__ import annotations

import numpy as np
import pytest

import tg_gb300 as tg
from oracle_lib import shade_render
from scenes import fuzz_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["rotated", "scaled", "sheared", "mirrored", "projective", "huge", "singular", "nan", "far"])
def test_shading_equals_the_oracle_for_any_matrix(ctx, oracle, kind):
    import torch
    s = fuzz_scene(31, n_objects=7, box=30.0, max_cpa=4)
    s.objects["lut_idx"] = 0
    rng = np.random.default_rng(7)
    m = s.objects["rotation"].reshape(7, 4, 4)   # m[object][column][row]
    if kind == "scaled":
        m[:, :3] *= np.float32(2.5)
    elif kind == "sheared":
        m[:, :3, :3] += rng.normal(size=(7, 3, 3)).astype(np.float32) * 0.3
    elif kind == "mirrored":
        m[:, 0] *= np.float32(-1.0)
    elif kind == "projective":
        m[:] = rng.normal(size=(7, 4, 4))
    elif kind == "huge":
        m[:, 1, :3] *= np.float32(1e-31)
    elif kind == "singular":
        m[:, 1] = m[:, 2]
    elif kind == "nan":
        m[::2, 0, 1] = np.nan
        m[1::2, 3, 0] = np.inf
    elif kind == "far":
        s.objects["translation"][::2] = 3e38
        s.objects["translation"][1::2] = 1e20
    view = tg.make_view((0.0, 5.0, -70.0), 0.1, float(np.pi), 1.1, 93, 61, 0.1, 300.0)
    n = 93 * 61
    words = (rng.integers(0, 1 << 24, n).astype(np.uint64) << np.uint64(40)) | \
            (rng.integers(0, len(s.cluster_pointers), n).astype(np.uint64) << np.uint64(9)) | \
            rng.integers(0, 512, n).astype(np.uint64)
    sc = ctx.upload(s)
    vis = torch.empty(n, dtype=torch.int64, device="cuda")
    ctx.vis_render(sc, view, [vis])
    ctx.sync()
    frame = vis.cpu().numpy().view(np.uint64)
    words[::2] = frame[::2]
    vis = torch.from_numpy(words.view(np.int64)).cuda()
    rgba = torch.empty(n * 4, dtype=torch.float32, device="cuda")
    for mode in (0, 8):
        torch.cuda.synchronize()
        ctx.shade(sc, view, vis, mode, rgba)
        ctx.sync()
        g = rgba.cpu().numpy().reshape(-1, 4)
        ref = shade_render(oracle, s, view, words, mode)
        same = (g.view(np.uint32) == ref.view(np.uint32)) | (np.isnan(g) & np.isnan(ref))
        assert same.all(), (kind, mode, int((~same).sum()))
    sc.close()
