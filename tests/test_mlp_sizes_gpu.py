"""Cache inference at every size where its tiles, groups and CTAs change: a
query's output does not depend on the batch it comes in, bit for bit, small
batches match the FP64 oracle within BF16 rounding (the tolerances of
test_mlp_gpu.py), and NaN or infinite inputs leave the other queries alone."""
from __future__ import annotations

import numpy as np
import pytest

import tg_gb300 as tg
from oracle_lib import OracleMlp
from test_mlp_gpu import batch, bf16_round

pytestmark = pytest.mark.gpu

SMS, GROUPS, TILE = 152, 6, 128


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, SMS * TILE - 1, SMS * TILE + 1, GROUPS * SMS * TILE - 7,
                               GROUPS * SMS * TILE + 1, 2 * GROUPS * SMS * TILE + 131])
def test_outputs_do_not_depend_on_the_batch(ctx, oracle, n):
    import torch
    cache = tg.Cache(ctx, seed=3)
    x, _ = batch(n, 5)
    odd = np.arange(n) % 11 == 4
    x[odd, np.arange(n)[odd] % 9] = np.where(np.arange(n)[odd] % 2 == 0, np.nan, np.inf)
    whole = torch.full((n + 8, 3), 7.0, dtype=torch.float32, device="cuda")
    dx = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    cache.infer(dx, whole)
    ctx.sync()
    y = whole.cpu().numpy()
    assert np.all(y[n:] == 7.0)
    for first in sorted({0, n // 3, max(0, n - 129)}):   # the same queries in other places of other batches
        m = min(n - first, 129)
        part = torch.empty((m, 3), dtype=torch.float32, device="cuda")
        sub = dx[first:first + m].clone()
        torch.cuda.synchronize()
        cache.infer(sub, part)
        ctx.sync()
        assert np.array_equal(part.cpu().numpy().view(np.uint32), y[first:first + m].view(np.uint32)), first
    assert ctx.device_error().code == 0
    if n <= 129:
        want = OracleMlp(oracle).forward(bf16_round(cache.get_weights()), x[~odd])
        scale = np.abs(want).mean()
        assert np.all(np.abs(y[:n][~odd] - want) <= 0.03 * np.abs(want) + 0.04 * scale)
    cache.close()


@pytest.mark.parametrize("n", [1, 127, 128, 129, SMS * TILE - 1, SMS * TILE + 1, 2 * SMS * TILE + 131])
def test_steps_back_to_back_equal_steps_with_a_wait_between(ctx, n):
    """A step's kernels read parameters and moments ahead of their wait for the
    kernel before: new batches every step, other work between the steps, and
    weights set between them change no bit against steps that run alone."""
    import torch
    batches = [tuple(torch.from_numpy(a).cuda() for a in batch(n, 20 + k)) for k in range(5)]
    out = torch.empty((64, 3), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    results = []
    for wait in (True, False, False):
        cache = tg.Cache(ctx, seed=7)
        w0 = cache.get_weights()
        for round_ in range(2):
            for k, (x, t) in enumerate(batches):
                cache.train_step(x, t, 5e-3)
                if k == 2:
                    cache.infer(x[:64].expand(64, 9).contiguous() if n == 1 else x[:64], out[:min(n, 64)] if n > 1 else out)
                if wait:
                    ctx.sync()
            if round_ == 0:
                results.append(cache.get_weights())
                cache.set_weights(w0)
        results.append(cache.get_weights())
        results.append(np.array([cache.last_loss()], np.float32))
        cache.close()
    assert ctx.device_error().code == 0
    for i in range(3):
        assert np.array_equal(results[i].view(np.uint32), results[3 + i].view(np.uint32))
        assert np.array_equal(results[i].view(np.uint32), results[6 + i].view(np.uint32))
    assert not np.array_equal(results[0], results[1])   # the moments went on
