"""A caller's choice of kernel variants holds in the calls that run its kind, in streamed calls
too, and leaves the others their own routes."""
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
