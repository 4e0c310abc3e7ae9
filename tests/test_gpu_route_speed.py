"""The rules that choose a kernel by a batch's size do not lose to the kernels that they pass by
on batches that are nothing but contacts (times of the two in turn, the best of several)."""
import numpy as np
import pytest

from ogx import workloads as W

pytestmark = pytest.mark.gpu


def contacts(n, points, apart=0.2):
    """n pairs of bodies of `points` points on a unit sphere, `apart` from one another."""
    g = np.random.default_rng(points)
    x = g.normal(size=(2 * n * points, 3))
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    c = np.zeros((2 * n, 3))
    d = g.normal(size=(n, 3))
    c[1::2] = apart * d / np.linalg.norm(d, axis=1, keepdims=True)
    x += np.repeat(c, points, axis=0)
    return W.Batch(x.astype(np.float32), np.arange(2 * n, dtype=np.int64) * points, np.full(2 * n, points, np.int32),
                   np.arange(2 * n, dtype=np.int32).reshape(-1, 2), "contacts")


def choose(ctx):
    """The caller's own choice of the context's variants (turns the size rules off)."""
    for kind in ("gjk", "epa"):
        for k, (lanes, blocks) in enumerate(ctx.kernel_choice()[kind]):
            ctx.set_kernel_choice(kind, k, lanes, blocks)


def best_ms(engine, b, ctxs, reps=30):
    import torch
    pairs = torch.from_numpy(b.pairs).cuda()
    pools = []
    for ctx in ctxs:
        pools.append(engine.Pool(ctx, b.counts))
        pools[-1].upload(b.coords)
    out, best = engine.Results(b.n_pairs, pairs.device), [1e9] * len(ctxs)
    for _ in range(reps):
        for i, (ctx, pool) in enumerate(zip(ctxs, pools)):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda.synchronize()
            with torch.cuda.stream(ctx.stream):
                e[0].record()
                engine.run(ctx, pool, pairs, engine.MODE_GJK_EPA, out)
                e[1].record()
            torch.cuda.synchronize()
            best[i] = min(best[i], e[0].elapsed_time(e[1]))
    return best


@pytest.mark.parametrize("n,points", [(8000, 16), (16000, 16), (24000, 32), (12000, 64)])
def test_contacts_of_a_medium_batch(engine, n, points):
    rule, tuned = engine.Context(0), engine.Context(0)
    choose(tuned)
    a, b = best_ms(engine, contacts(n, points), [rule, tuned])
    assert a < 1.2 * b, (a, b)


@pytest.mark.parametrize("n,points", [(2500, 200), (2500, 400), (4000, 400)])
def test_few_contacts_of_large_bodies(engine, n, points):
    rule, narrow = engine.Context(0), engine.Context(0)
    choose(narrow)
    a, b = best_ms(engine, contacts(n, points, 1.0), [rule, narrow])
    assert a < 1.1 * b, (a, b)


@pytest.mark.parametrize("points", [300, 400, 512])
def test_contacts_of_large_bodies(engine, points):
    """257 to 512 points, more contacts than the rules for medium batches take."""
    rule, narrow, wide = (engine.Context(0) for _ in range(3))
    for ctx, lanes in ((narrow, 8), (wide, 16)):
        choose(ctx)
        ctx.set_kernel_choice("epa", 5, lanes, 5 << 8)
    a, b, c = best_ms(engine, contacts(30000, points, 1.0), [rule, narrow, wide], reps=10)
    assert a < 1.2 * min(b, c), (a, b, c)
