"""EPA's kernels of medium batches and of large bodies choose their width by the contacts that a
bucket holds: the same bits as the variants with a fixed width, on both sides of each limit."""
import numpy as np
import pytest

from ogx import workloads as W
from test_gpu_route_speed import choose, contacts

pytestmark = pytest.mark.gpu


def twins(n, points):
    """n pairs of bodies of the same `points` points on a unit sphere, a little apart: all of them
    are contacts."""
    b = contacts(n, points)
    x = b.coords.reshape(n, 2, points, 3)
    x[:, 1] = x[:, 0] + np.float32(0.03) * np.random.default_rng(n).normal(size=(n, 1, 3)).astype(np.float32)
    return b


def _with_contacts(engine, few, rest, want):
    """The first pairs of `few` and all of `rest`, as many of the former as make exactly `want`
    contacts for the bucket kernels (a few are found only by the refinement)."""
    import torch
    ctx = engine.Context(0)
    bodies = W.Batch(np.concatenate([few.coords, rest.coords]),
                     np.concatenate([few.offsets, rest.offsets + few.coords.shape[0]]),
                     np.concatenate([few.counts, rest.counts]), None, "joined")
    pool = engine.Pool(ctx, bodies.counts)
    pool.upload(bodies.coords)
    lo, hi = want, few.n_pairs
    while True:
        m = (lo + hi) // 2
        bodies.pairs = np.concatenate([few.pairs[:m], rest.pairs + few.n_bodies]).astype(np.int32)
        engine.run(ctx, pool, torch.from_numpy(bodies.pairs).cuda(), engine.MODE_GJK_EPA)
        ctx.synchronize()
        n = sum(ctx.work_counts()["epa"])
        if n == want:
            return bodies
        assert lo < hi, (want, n)
        lo, hi = (m + 1, hi) if n < want else (lo, m - 1)


def _same(engine, b, mode):
    import torch
    pairs, out = torch.from_numpy(b.pairs).cuda(), []
    for chosen in (False, True):
        ctx = engine.Context(0)
        if chosen:
            choose(ctx)
        pool = engine.Pool(ctx, b.counts)
        pool.upload(b.coords)
        res = None
        if mode == engine.MODE_EPA:
            res = engine.run(ctx, pool, pairs, engine.MODE_GJK, engine.Results(b.n_pairs, pairs.device))
        out.append(engine.run(ctx, pool, pairs, mode, res).to_host())
        ctx.synchronize()
    for k in ("dist", "normal", "status", "simplex"):
        assert out[0][k].tobytes() == out[1][k].tobytes(), k


@pytest.mark.parametrize("points,limit", [(6, 1000), (24, 1000), (60, 1000), (100, 1000), (200, 2000), (400, 3000),
                                          (600, 2000)])
@pytest.mark.parametrize("above", [0, 1])
def test_medium_batches(engine, points, limit, above):
    # `limit + above` contacts of this size among separated pairs of small bodies
    b = _with_contacts(engine, twins(limit + 200, points), contacts(3000, 5, apart=4.0), limit + above)
    _same(engine, b, engine.MODE_GJK_EPA)
    _same(engine, b, engine.MODE_EPA)


@pytest.mark.parametrize("share", [0.3, 0.45])
def test_large_bodies(engine, share):
    n = 32000  # the limit is 3/8 of them
    b = _with_contacts(engine, twins(int(share * n) + 300, 300), contacts(n - int(share * n), 5, apart=4.0),
                       int(share * n))
    assert b.n_pairs > 24576 and (8 * int(share * n) > 3 * b.n_pairs) == (share > 0.4)
    _same(engine, b, engine.MODE_GJK_EPA)


def test_large_posed_bodies(engine, twin):
    """Bodies of 257 to 512 points in their own frames, nearly all of the pairs in contact."""
    from ogx import serving
    scene = W.serving_scene(seed=5, n_bodies=300, lo=300, hi=500, half=0.5)
    xf = scene.transforms(0)
    g = np.random.default_rng(1)
    pairs = g.integers(0, 300, (3000, 2)).astype(np.int32)
    pairs = np.ascontiguousarray(pairs[pairs[:, 0] != pairs[:, 1]])
    with serving.Server(scene.counts, scene.local, warm_start=False, fused_transform=True) as srv:
        res = srv.wait(srv.submit(srv.set_transforms(xf), pairs))
        dist = np.array(res.dist)
    h = twin.run(W.Batch(scene.local, scene.offsets, scene.counts, pairs, "serving"), xf=xf)
    assert (h["dist"] < 0).mean() > 0.9
    assert (dist == h["dist"]).mean() > 0.995
