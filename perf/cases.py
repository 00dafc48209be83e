"""Performance cases: what a user of the library has it do, through its public entry points.

Every case is a dict of plain values.  `prepare` makes the inputs from a seed
(scenes, cameras, rays and batches differ from seed to seed) together with the
context, scene, SVO, graph or cache that a program keeps; `run` makes one pass
and returns its outputs.  Scenes are the synthetic generator's, with the sizes
of the benchmark and the tests: one Bernoulli cloud, or many value-noise
objects of 2..16 clusters per axis with the density of the 512-object scene.
The contexts of all states run on one torch stream, as in a program that mixes
the library with its own torch work.

kinds
  frame    tgx_vis_render (and tgx_shade): the engine's frame
  batch    a captured frame graph over several scenes and uneven views, new cameras each frame
  host     tgx_vis_render_host into pinned memory: a caller that reads every frame back
  build    tgx_svo_build, then the first lit preview frame over it (a level load)
  update   objects move: tgx_scene_set_objects + tgx_svo_update and a lit preview frame, there and back
  trace    tgx_svo_trace of a ray batch
  gi       tgx_gi_render: plain bounce lighting of a visibility buffer
  cached   tgx_gi_render_cached: a frame that trains the cache, or one that only uses it (with the blend)
  infer    tgx_cache_infer
  train    tgx_cache_train_step, several steps, then the weights to the host
"""
import math
import random

import numpy as np
import torch

import tg_gb300 as tg

RESOLUTIONS = ((320, 240), (640, 480), (1280, 720), (1920, 1080), (3840, 2160))
PREVIEW = (480, 270)          # the lit preview frame of the build and update cases
FOV = math.pi / 3
_STREAM = []


def listed():
    return [
        # the smallest call: one 32^3 object at 256x256, where launches and latency are all there is
        dict(name="frame-cloud-256", kind="frame", objects=0, cpa=4, w=256, h=256, tile_w=16, tile_h=16, shade=False),
        # the ordinary frame: the 512-object scene at 1080p, visibility and direct shading
        dict(name="frame-512-1080p", kind="frame", objects=512, cpa=16, w=1920, h=1080, tile_w=8, tile_h=8, shade=True),
        # many cameras and scenes of uneven size in one graph, up to 4K views
        dict(name="batch-20-views", kind="batch", views=16, scenes=4, mix=3, tile_w=8, tile_h=8),
        # the frame read back into host memory
        dict(name="host-512-1080p", kind="host", objects=512, cpa=16, w=1920, h=1080, tile_w=8, tile_h=8),
        # a level load: the 4096^3 SVO with materials
        dict(name="build-512", kind="build", objects=512, cpa=16, log2=12),
        # 8 of 512 objects move every frame
        dict(name="update-512-8", kind="update", objects=512, cpa=16, log2=12, moved=8),
        # ray queries of an engine (physics, audio, picking)
        dict(name="trace-1m", kind="trace", objects=512, cpa=16, log2=12, rays=1000003),
        # plain bounce lighting of the 1080p frame
        dict(name="gi-1080p-4spp", kind="gi", objects=512, cpa=16, w=1920, h=1080, spp=4, bounces=1),
        # the learned cache's frame with its configured training budget
        dict(name="cached-train-1080p", kind="cached", objects=512, cpa=16, w=1920, h=1080, spp=2, n_train=65536,
             train_spp=16, steps=16, n_train_primary=131072),
        # the cache used without training (an odd window size), with the pixel-point blend
        dict(name="cached-use-853x479", kind="cached", objects=512, cpa=16, w=853, h=479, spp=3, n_train=0,
             train_spp=0, steps=0, n_train_primary=0),
        # the network alone: a frame's queries, and a frame's training
        dict(name="infer-1m", kind="infer", n=1 << 20),
        dict(name="train-16x4096", kind="train", n=4096, steps=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "batch", "host", "build", "update", "trace", "gi", "cached", "infer", "train"])
    objects = rng.choice([0, _log(rng, 8, 1024), _log(rng, 32, 512)])
    cpa = rng.randint(2, 8) if objects == 0 else rng.randint(3, 16)
    tile_w, tile_h = rng.choice([(8, 8), (8, 8), (16, 8), (8, 16), (16, 16), (32, 8)])
    w = _log(rng, 96, 1920)
    h = max(1, int(w * rng.uniform(0.45, 1.0)))
    h = min(h, 1080)
    if kind in ("frame", "host"):
        c = dict(kind=kind, objects=objects, cpa=cpa, w=w, h=h, tile_w=tile_w, tile_h=tile_h)
        return dict(c, shade=rng.random() < 0.5) if kind == "frame" else c
    if kind == "batch":
        return dict(kind=kind, views=rng.randint(2, 14), scenes=rng.randint(0, 4), mix=rng.randrange(1 << 20),
                    tile_w=tile_w, tile_h=tile_h)
    objects = objects or _log(rng, 16, 512)
    cpa = max(cpa, 3)
    log2 = rng.choice([10, 11, 12])
    if kind == "build":
        return dict(kind=kind, objects=min(objects, 512), cpa=cpa, log2=log2)
    if kind == "update":
        objects = min(objects, 512)
        return dict(kind=kind, objects=objects, cpa=cpa, log2=log2, moved=min(objects, _log(rng, 1, 32)))
    if kind == "trace":
        return dict(kind=kind, objects=min(objects, 512), cpa=cpa, log2=log2, rays=_log(rng, 1, 1 << 20))
    if kind == "gi":
        bounces = rng.choice([1, 1, 2, 3])
        spp = max(1, min(_log(rng, 1, 16), int(4 * 1920 * 1080 / (w * h * bounces))))
        return dict(kind=kind, objects=min(objects, 512), cpa=cpa, w=w, h=h, spp=spp, bounces=bounces)
    if kind == "cached":
        spp = rng.choice([1, 2, 2, 3])
        if rng.random() < 0.5 or w * h * spp > 2 * 1920 * 1080:
            n_train, steps = _log(rng, 1024, 65536), rng.choice([1, 4, 8, 16])
            return dict(kind=kind, objects=min(objects, 512), cpa=cpa, w=w, h=h, spp=min(spp, 2), n_train=n_train,
                        train_spp=rng.choice([8, 16]), steps=steps, n_train_primary=rng.choice([0, 2 * n_train]))
        return dict(kind=kind, objects=min(objects, 512), cpa=cpa, w=w, h=h, spp=spp, n_train=0, train_spp=0, steps=0,
                    n_train_primary=0)
    if kind == "infer":
        return dict(kind=kind, n=_log(rng, 1, 1 << 20))
    return dict(kind=kind, n=_log(rng, 64, 65536), steps=rng.randint(1, 16))


# ---- inputs ------------------------------------------------------------------

def _context(case):
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return tg.Context(torch.cuda.current_device(), stream=_STREAM[0].cuda_stream,
                      tile=(case.get("tile_w", 8), case.get("tile_h", 8)))


def _half(objects):
    """Half the side of the box that keeps the 512-object scene's density."""
    return 1024.0 * (objects / 512.0) ** (1.0 / 3.0)


def _scene(ctx, objects, cpa, seed):
    if objects == 0:   # one cloud in front of a camera at the origin
        return ctx.generate_scene(0, 1, cpa, cpa, seed, bernoulli_p=0.3, translation=(0.0, 0.0, 16.0 * cpa), n_luts=32)
    half = _half(objects)
    return ctx.generate_scene(1, objects, 2, max(2, cpa), seed, noise_period=64.0, noise_threshold=0.5,
                              box_min=(-half,) * 3, box_max=(half,) * 3, n_luts=32)


def _view(objects, w, h, rng):
    if objects == 0:
        return tg.make_view((0.0, 0.0, 0.0), 0.0, math.pi, FOV, w, h, 0.1, 256.0)
    half = _half(objects)
    return tg.make_view(tuple(float(x) for x in rng.uniform(-0.25 * half, 0.25 * half, 3)), float(rng.uniform(-0.3, 0.3)),
                        float(rng.uniform(0.0, 2.0 * math.pi)), FOV, w, h, 0.1, 4.0 * half)


def _svo(ctx, scene, objects, log2):
    half = float(1 << (log2 - 1))
    return ctx.svo_build(scene, (-half, -half, -half), log2)


def _pixels(w, h):
    return torch.empty(w * h, dtype=torch.int64, device="cuda")


def _rgb(w, h):
    return torch.empty(w * h * 3, dtype=torch.float32, device="cuda")


def _weights(seed):
    """He-uniform weights in the library's flat order (W0 [64][216], W1..W3 [64][64], W4 [3][64])."""
    rng = np.random.default_rng(seed)
    n0, n1 = 64 * 216, 3 * 64 * 64 + 3 * 64
    b = np.concatenate([np.full(n0, math.sqrt(6.0 / 216)), np.full(n1, math.sqrt(6.0 / 64))])
    return (rng.uniform(-1.0, 1.0, n0 + n1) * b).astype(np.float32)


def _queries(n, seed):
    """Network inputs (position in the unit box, unit normal and direction) and a smooth target."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.cat([torch.rand((n, 3), generator=g, device="cuda"),
                   torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1),
                   torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)], dim=1)
    t = 0.3 + 0.2 * torch.sin(4.0 * x[:, :3]) + 0.1 * x[:, 3:6] ** 2
    return x.contiguous(), t.contiguous()


def _batch_jobs(case):
    """[(objects, [(w, h), ...]), ...]: the views of the 512-object scene, then one view per further scene."""
    rng = random.Random(case["mix"])
    jobs = [(512, [rng.choice(RESOLUTIONS) for _ in range(case["views"])])]
    for _ in range(case["scenes"]):
        jobs.append((_log(rng, 32, 2048), [rng.choice(RESOLUTIONS)]))
    return jobs


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    s = dict(case=case, kind=kind, ctx=_context(case))
    ctx = s["ctx"]
    if kind in ("frame", "host"):
        w, h = case["w"], case["h"]
        s["scene"] = _scene(ctx, case["objects"], case["cpa"], seed + 1)
        s["view"] = _view(case["objects"], w, h, rng)
        if kind == "host":
            s["out"] = torch.empty(w * h, dtype=torch.int64, pin_memory=True).numpy()
        else:
            s["vis"] = _pixels(w, h)
            s["rgba"] = torch.empty((w * h, 4), dtype=torch.float32, device="cuda") if case["shade"] else None
    elif kind == "batch":
        s["jobs"] = []
        for k, (objects, sizes) in enumerate(_batch_jobs(case)):
            views = np.concatenate([_view(objects, w, h, rng) for w, h in sizes])
            s["jobs"].append((_scene(ctx, objects, 16, seed + 1 + k), views, [_pixels(w, h) for w, h in sizes]))
        s["graph"] = ctx.frame_graph(s["jobs"])
        # the cameras of the frame that run() renders
        s["views"] = [np.concatenate([_view(objects, w, h, rng) for w, h in sizes]) for objects, sizes in _batch_jobs(case)]
    elif kind in ("infer", "train"):
        s["cache"] = tg.Cache(ctx, seed=1)
        s["cache"].set_weights(_weights(seed))
        s["x"], s["t"] = _queries(case["n"] * case.get("steps", 1), seed)
        s["y"] = torch.empty((case["n"], 3), dtype=torch.float32, device="cuda")
    else:
        objects = case["objects"]
        s["scene"] = _scene(ctx, objects, case["cpa"], seed + 1)
        w, h = (case["w"], case["h"]) if kind in ("gi", "cached") else PREVIEW
        s["view"] = _view(objects, w, h, rng)
        s["vis"], s["rgb"] = _pixels(w, h), _rgb(w, h)
        if kind != "build":
            s["svo"] = _svo(ctx, s["scene"], objects, case.get("log2", 12))
        if kind == "update":
            s["vis2"], s["rgb2"] = _pixels(w, h), _rgb(w, h)
            here = s["scene"].download().objects[:case["moved"]]
            there = here.copy()
            there["translation"] += rng.uniform(-40.0, 40.0, there["translation"].shape).astype(np.float32)
            s["poses"] = (there, here)
        elif kind == "trace":
            n, half = case["rays"], min(_half(objects), float(1 << (case["log2"] - 1)))
            g = torch.Generator(device="cuda").manual_seed(seed)
            s["o"] = (torch.rand((n, 3), generator=g, device="cuda") * 2.0 - 1.0) * half
            s["d"] = torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)
            s["t"] = torch.empty(n, dtype=torch.float32, device="cuda")
            s["voxel"] = torch.empty((n, 3), dtype=torch.int32, device="cuda")
        elif kind in ("gi", "cached"):
            torch.cuda.synchronize()
            ctx.vis_render(s["scene"], s["view"], [s["vis"]])
        s["gi"] = tg.gi_params(spp=case.get("spp", 2), bounces=case.get("bounces", 2 if kind == "cached" else 1),
                               seed=seed + 2, max_steps=256)
        if kind == "cached":
            half = _half(objects) + 160.0
            s["cache"] = tg.Cache(ctx, seed=seed + 3)
            s["w0"] = _weights(seed)
            s["cache"].set_weights(s["w0"])
            use = case["n_train"] == 0
            s["cp"] = tg.cache_gi_params((-half,) * 3, (half,) * 3, n_train=case["n_train"], train_spp=case["train_spp"],
                                         train_steps=case["steps"], lr=5e-4, primary_weight=1.0 if use else 0.0,
                                         n_train_primary=case["n_train_primary"])
    torch.cuda.synchronize()
    ctx.sync()
    return s


# ---- one pass ----------------------------------------------------------------

def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "frame":
        ctx.vis_render(s["scene"], s["view"], [s["vis"]])
        if s["rgba"] is None:
            return s["vis"]
        ctx.shade(s["scene"], s["view"], s["vis"], 0, s["rgba"])
        return s["vis"], s["rgba"]
    if kind == "host":
        ctx.vis_render_host(s["scene"], s["view"], [s["out"]])
        return s["out"]
    if kind == "batch":
        for k, views in enumerate(s["views"]):
            s["graph"].set_views(k, views)
        s["graph"].launch()
        return [o for _, _, outs in s["jobs"] for o in outs]
    if kind == "build":
        svo = _svo(ctx, s["scene"], s["case"]["objects"], s["case"]["log2"])
        ctx.vis_render(s["scene"], s["view"], [s["vis"]])
        ctx.gi_render(s["scene"], svo, s["view"], s["vis"], s["gi"], s["rgb"])
        i = svo.info()
        svo.close()
        return {"blocks": int(i.n_blocks), "nonempty": int(i.n_nonempty_blocks), "pairs": int(i.n_pairs),
                "vis": s["vis"], "rgb": s["rgb"]}
    if kind == "update":
        moved = []
        for objs, vis, rgb in zip(s["poses"], (s["vis"], s["vis2"]), (s["rgb"], s["rgb2"])):
            s["scene"].set_objects(0, objs)
            moved.append(s["svo"].update(s["scene"]))
            ctx.vis_render(s["scene"], s["view"], [vis])
            ctx.gi_render(s["scene"], s["svo"], s["view"], vis, s["gi"], rgb)
        return {"moved": moved, "vis": [s["vis"], s["vis2"]], "rgb": [s["rgb"], s["rgb2"]]}
    if kind == "trace":
        s["svo"].trace(s["o"], s["d"], s["t"], s["voxel"], max_steps=256)
        return s["t"], s["voxel"]
    if kind == "gi":
        ctx.gi_render(s["scene"], s["svo"], s["view"], s["vis"], s["gi"], s["rgb"])
        return s["rgb"]
    if kind == "cached":
        if s["case"]["n_train"]:   # a cut to a known state of the cache, then the frame that trains it
            s["cache"].set_weights(s["w0"])
        ctx.gi_render_cached(s["scene"], s["svo"], s["cache"], s["view"], s["vis"], s["gi"], s["cp"], s["rgb"])
        return (s["rgb"], s["cache"].get_weights()) if s["case"]["n_train"] else s["rgb"]
    if kind == "infer":
        s["cache"].infer(s["x"], s["y"])
        return s["y"]
    n = s["case"]["n"]
    for k in range(s["case"]["steps"]):
        s["cache"].train_step(s["x"][k * n:(k + 1) * n], s["t"][k * n:(k + 1) * n], 1e-2)
    return s["cache"].get_weights()


# ---- what a pass cannot do without -------------------------------------------

def _clusters(objects, cpa):
    return cpa ** 3 if objects == 0 else objects * ((2 + max(2, cpa)) / 2.0) ** 3


def _vis_work(objects, cpa, pixels):
    """8 bytes out per pixel, every object and cluster pointer once, and the bitmask and pointer of the clusters
    in view (about one in ten of a scene around the camera); a ray set-up and about two DDA steps per pixel."""
    n = _clusters(objects, cpa)
    seen = n if objects == 0 else 0.1 * n
    return 8.0 * pixels + 96.0 * max(objects, 1) + 4.0 * n + 72.0 * seen, 60.0 * pixels


def _ray_work(rays):
    """24 bytes in and 16 out per ray, about 45 traversal steps of 20 operations."""
    return 40.0 * rays, 900.0 * rays


def _gi_work(pixels, spp, bounces):
    """The visibility words in and RGB out; about a third of the pixels see geometry and trace, per sample and
    bounce, a bounce ray and half a shadow ray (what a ray reads stays on chip: only its operations count)."""
    rays = pixels / 3.0 * (1.0 + 1.5 * spp * bounces)
    return 20.0 * pixels, _ray_work(rays)[1]


FWD_FLOPS = 2.0 * (216 * 64 + 3 * 64 * 64 + 64 * 3)
TRAIN_FLOPS = 2.0 * FWD_FLOPS + 2.0 * (3 * 64 * 64 + 64 * 3)


def work(case):
    kind = case["kind"]
    if kind in ("frame", "host"):
        px = case["w"] * case["h"]
        b, f = _vis_work(case["objects"], case["cpa"], px)
        if case.get("shade"):
            b, f = b + 24.0 * px, f + 80.0 * px
    elif kind == "batch":
        b = f = 0.0
        for objects, sizes in _batch_jobs(case):
            for w, h in sizes:
                vb, vf = _vis_work(objects, 16, w * h)
                b, f = b + vb, f + vf
    elif kind in ("build", "update"):
        n = _clusters(case["objects"], case["cpa"])
        if kind == "update":   # two frames, each with the moved objects' clusters in both poses
            n *= 4.0 * case["moved"] / case["objects"]
        px = PREVIEW[0] * PREVIEW[1] * (2 if kind == "update" else 1)
        gb, gf = _gi_work(px, 2, 1)
        vb, vf = _vis_work(case["objects"], case["cpa"], px)
        # every cluster's bits and materials in; half of its 512 voxels' bits and material codes out
        b, f = n * (64 + 512 + 64 + 512 * 2) + gb + vb, n * 512 * 30.0 + gf + vf
    elif kind == "trace":
        b, f = _ray_work(case["rays"])
    elif kind == "gi":
        b, f = _gi_work(case["w"] * case["h"], case["spp"], case["bounces"])
    elif kind == "cached":
        px = case["w"] * case["h"]
        b, f = _gi_work(px, case["spp"], 1)
        queries = px / 3.0 * case["spp"] * 0.5 + (0.0 if case["n_train"] else px / 3.0)
        rays = case["n_train"] * case["train_spp"] * 1.5
        trained = (case["n_train"] + case["n_train_primary"]) if case["steps"] else 0
        f += queries * FWD_FLOPS + _ray_work(rays)[1] + trained * TRAIN_FLOPS
    elif kind == "infer":
        b, f = 48.0 * case["n"] + 53000.0, FWD_FLOPS * case["n"]
    else:
        n = case["n"] * case["steps"]
        b, f = 48.0 * n + 53000.0 * 10 * case["steps"], TRAIN_FLOPS * n
    return {"bytes": b, "flops": f}


# ---- the network in 64 bits --------------------------------------------------

def _layers(w):
    out, at = [], 0
    for rows, cols in ((64, 216), (64, 64), (64, 64), (64, 64), (3, 64)):
        out.append(w[at:at + rows * cols].reshape(rows, cols))
        at += rows * cols
    return out


def _encode(x):
    a = x.double()[:, :, None] * (math.pi * 2.0 ** torch.arange(12, dtype=torch.float64, device=x.device))
    return torch.stack((torch.sin(a), torch.cos(a)), dim=3).reshape(x.shape[0], 216)


def _forward(w, x):
    h = [_encode(x)]
    for l, m in enumerate(_layers(w)):
        z = h[-1] @ m.T
        h.append(z.clamp_min(0.0) if l < 4 else z)
    return h


def exact(case, seed):
    """The network's outputs and trained weights in 64 bits; nothing for buffers of words and for path-traced frames,
    where a last bit decides which voxel a ray meets."""
    if case["kind"] not in ("infer", "train"):
        return None
    w = torch.from_numpy(_weights(seed)).cuda().double()
    n = case["n"]
    x, t = _queries(n * case.get("steps", 1), seed)
    if case["kind"] == "infer":
        return torch.cat([_forward(w, p)[-1] for p in x.split(1 << 17)])
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    for k in range(case["steps"]):
        g = [torch.zeros_like(l) for l in _layers(w)]
        for p, q in zip(x[k * n:(k + 1) * n].split(1 << 15), t[k * n:(k + 1) * n].split(1 << 15)):
            h = _forward(w, p)
            y = h[-1]
            d = 2.0 * (y - q.double()) / (y * y + 0.01) / (3.0 * n)   # relative L2, its denominator held fixed
            for l in range(4, -1, -1):
                g[l] += d.T @ h[l]
                if l:
                    d = (d @ _layers(w)[l]) * (h[l] > 0.0)
        g = torch.cat([a.reshape(-1) for a in g])
        m, v = 0.9 * m + 0.1 * g, 0.99 * v + 0.01 * g * g
        w = w - 1e-2 * (m / (1.0 - 0.9 ** (k + 1))) / (torch.sqrt(v / (1.0 - 0.99 ** (k + 1))) + 1e-15)
    return w.cpu().numpy()
