"""Frames one after the other on one context: view counts on both sides of what
the first kernel takes as its argument, counters that take turns, a frame whose
bins overflow, a frame graph and a frame captured by the caller between them.
Every buffer and every statistic equals those of a context of its own."""
from __future__ import annotations

import numpy as np
import pytest

import tg_gb300 as tg
from scenes import fuzz_scene

pytestmark = pytest.mark.gpu


def cameras(n, seed):
    rng = np.random.default_rng(seed)
    return [tg.make_view(tuple(rng.uniform(-30, 30, 3) + (0, 0, -60)), 0.1, float(np.pi) + rng.uniform(-0.3, 0.3), 1.1,
                         int(rng.integers(20, 90)), int(rng.integers(20, 70)), 0.1, 300.0) for _ in range(n)]


def outputs(views):
    import torch
    return [torch.full((int(np.atleast_1d(v)["width"][0]) * int(np.atleast_1d(v)["height"][0]),), 7, dtype=torch.int64, device="cuda") for v in views]


def stats(ctx):
    s = ctx.vis_stats()
    return s.visible_clusters, s.bin_entries, s.tiles, s.dda_overruns


def render(ctx, sc, views):
    import torch
    outs = outputs(views)
    torch.cuda.synchronize()
    ctx.vis_render(sc, np.concatenate([np.atleast_1d(v) for v in views]), outs)
    return outs


@pytest.mark.parametrize("flags", [0, tg.FLAG_MIN_BIN_CAPACITY])
def test_frames_in_turn_equal_frames_alone(flags):
    s = fuzz_scene(51, n_objects=9, box=30.0, max_cpa=3)
    counts = [1, 8, 9, 1, 1, 40, 8, 2, 9, 1]
    frames = [cameras(n, k) for k, n in enumerate(counts)]
    want = []
    for views in frames:
        with tg.Context(0, tile=(8, 8), flags=flags) as ctx:
            sc = ctx.upload(s)
            outs = render(ctx, sc, views)
            st = stats(ctx)
            want.append(([o.cpu().numpy() for o in outs], st))
            sc.close()
    with tg.Context(0, tile=(8, 8), flags=flags) as ctx:
        sc = ctx.upload(s)
        for read_stats in (True, False):           # with and without a wait after each frame
            got = []
            for views in frames:
                outs = render(ctx, sc, views)
                got.append((outs, stats(ctx) if read_stats else None))
            last = stats(ctx)
            for (outs, st), (w_outs, w_st) in zip(got, want):
                assert all(np.array_equal(o.cpu().numpy(), w) for o, w in zip(outs, w_outs))
                assert st is None or st == w_st
            assert last == want[-1][1]
        assert ctx.device_error().code == 0
        sc.close()


def test_frames_between_a_frame_graphs_launches():
    s = fuzz_scene(52, n_objects=9, box=30.0, max_cpa=3)
    views, other = cameras(3, 1), cameras(2, 2)
    with tg.Context(0, tile=(8, 8)) as ctx:
        sc = ctx.upload(s)
        w_views = [o.cpu().numpy() for o in render(ctx, sc, views)]
        w_other = [o.cpu().numpy() for o in render(ctx, sc, other)]
        outs = outputs(views)
        graph = ctx.frame_graph([(sc, np.concatenate([np.atleast_1d(v) for v in views]), outs)])
        for _ in range(3):
            for o in outs:
                o.fill_(9)
            import torch
            torch.cuda.synchronize()
            graph.launch()
            alone = render(ctx, sc, other)
            ctx.sync()
            assert all(np.array_equal(o.cpu().numpy(), w) for o, w in zip(outs, w_views))
            assert all(np.array_equal(o.cpu().numpy(), w) for o, w in zip(alone, w_other))
        graph.close()
        sc.close()


def test_frames_between_replays_of_a_captured_frame():
    import torch
    s = fuzz_scene(52, n_objects=9, box=30.0, max_cpa=3)
    (view,), other = cameras(1, 3), cameras(2, 4)
    stream = torch.cuda.Stream()
    with tg.Context(0, stream=stream.cuda_stream, tile=(8, 8)) as ctx:
        sc = ctx.upload(s)
        w_other = [o.cpu().numpy() for o in render(ctx, sc, other)]
        for _ in range(2):
            (out,) = render(ctx, sc, [view])
            ctx.sync()
        want = out.cpu().numpy()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            ctx.vis_render(sc, view, [out])
        for k in range(4):
            out.fill_(3)
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                graph.replay()
            frames = [render(ctx, sc, other) for _ in range(k)]
            ctx.sync()
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), want)
            for f in frames:
                assert all(np.array_equal(o.cpu().numpy(), w) for o, w in zip(f, w_other))
        sc.close()
