"""A caller's choice of kernel variants holds in the calls that run its kind, in streamed calls
too, and leaves the others their own routes."""
import os
import subprocess
import sys

import numpy as np
import pytest

from ogx import workloads as W

pytestmark = pytest.mark.gpu


def _set(ctx, kind):
    for k, (lanes, blocks) in enumerate(ctx.kernel_choice()[kind]):
        ctx.set_kernel_choice(kind, k, lanes, blocks)


def _launches(engine, ctx, b, mode):
    import torch
    pool = engine.Pool(ctx, b.counts)
    pool.upload(b.coords)
    pairs = torch.from_numpy(b.pairs).cuda()
    res = engine.run(ctx, pool, pairs, engine.MODE_GJK, engine.Results(b.n_pairs, pairs.device))
    if mode != engine.MODE_GJK:
        engine.run(ctx, pool, pairs, mode, res)
    ctx.synchronize()
    return ctx.last_launches


@pytest.mark.parametrize("kind", ["gjk", "epa"])
def test_a_choice_concerns_its_own_kind(engine, kind):
    b = W.powerlaw(seed=8, n_pairs=500)
    ctx = engine.Context(0)
    _set(ctx, kind)
    assert (_launches(engine, ctx, b, engine.MODE_GJK) == 1) == (kind == "epa")
    assert (_launches(engine, ctx, b, engine.MODE_EPA) == 1) == (kind == "gjk")
    assert _launches(engine, ctx, b, engine.MODE_GJK_EPA) > 1


def test_streamed_calls_take_the_choice(engine):
    b = W.powerlaw(seed=9, n_pairs=2000)
    launches, out = [], []
    for chosen in (False, True):
        ctx = engine.Context(0)
        if chosen:
            _set(ctx, "gjk")
            _set(ctx, "epa")
        pool = engine.Pool(ctx, b.counts)
        out.append(engine.streamed(ctx, pool, np.ascontiguousarray(b.coords), b.pairs, chunks=4))
        launches.append(ctx.last_launches)
    # (a chunk is one launch by default, and at least a kernel per bucket and kind otherwise)
    assert launches[0] <= 8 and launches[1] >= 4 * 14, launches
    for k in ("dist", "normal", "status", "simplex"):
        assert out[0][k].tobytes() == out[1][k].tobytes(), k


AUTOTUNE = """
import sys
sys.path[:0] = {path!r}
import torch
import test_gpu_route_speed as R
from ogx import engine
b = R.contacts(12000, 32)
tuned, chosen = engine.Context(0), engine.Context(0)
pool = engine.Pool(tuned, b.counts)
pool.upload(b.coords)
picked = tuned.autotune(pool, torch.from_numpy(b.pairs).cuda(), reps=3)
for kind in ("gjk", "epa"):
    for k, (lanes, blocks) in enumerate(picked[kind]):
        chosen.set_kernel_choice(kind, k, lanes, blocks)
later = engine.Context(0)
times = R.best_ms(engine, b, [tuned, later, chosen])
small = R.contacts(500, 32)
pool = engine.Pool(later, small.counts)
pool.upload(small.coords)
engine.run(later, pool, torch.from_numpy(small.pairs).cuda())
print(*times, later.last_launches)
"""


def test_calls_take_what_the_autotuner_kept(engine):
    """At the size that it was given, in the context and in later ones; smaller calls keep their
    route.  In a process of its own: the picks stay for the process."""
    code = AUTOTUNE.format(path=[os.path.dirname(os.path.abspath(__file__))] + sys.path)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-1000:]
    tuned, later, chosen, launches = (float(x) for x in r.stdout.split())
    assert tuned < 1.08 * chosen and later < 1.08 * chosen, (tuned, later, chosen)
    assert launches == 1


@pytest.mark.parametrize("n", [500, 3000])
def test_timing_leaves_the_route_alone(engine, n):
    import torch
    b = W.powerlaw(seed=10, n_pairs=n)
    ctx = engine.Context(0)
    pool = engine.Pool(ctx, b.counts)
    pool.upload(b.coords)
    pairs = torch.from_numpy(b.pairs).cuda()
    want = engine.run(ctx, pool, pairs).to_host()
    launches = ctx.last_launches
    ctx.set_timing(True)
    got = engine.run(ctx, pool, pairs).to_host()
    times = ctx.kernel_times()
    assert ctx.last_launches == launches
    assert (len(times) == 1) == (launches == 1) and all(t > 0 for _, t in times), times
    ctx.set_timing(False)
    ctx.set_stage_timeline(True)
    engine.run(ctx, pool, pairs)
    stages = ctx.stage_timeline()
    assert ctx.last_launches == launches and stages[-1][0] == "end" and stages[-1][1] > 0
    assert got["dist"].tobytes() == want["dist"].tobytes()
