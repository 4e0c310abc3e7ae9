"""A caller's choice of kernel variants holds in the calls that run its kind
and leaves the others their own routes."""
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
