"""Small batches run the whole pipeline with one warp per pair, larger ones the bucket
kernels, and between the two EPA takes a warp per contact: the same functions on other
teams, so the results are the bucket kernels' bit for bit, on both sides of every line
where the route changes."""
import numpy as np
import pytest

from ogx import workloads as W

pytestmark = pytest.mark.gpu


def _batch(n):
    """n pairs of every kind: power-law sizes up to 1024 points (capacity spills, every
    bucket) and the stress set (FP64 continuations, certified re-runs, late contacts)."""
    a, b = W.powerlaw(seed=70 + n, n_pairs=max(1, n // 2)), W.stress(seed=71 + n, n_pairs=max(3, n - n // 2))
    pairs = np.concatenate([a.pairs, b.pairs + a.n_bodies]).astype(np.int32)
    rng = np.random.default_rng(n)
    pairs = pairs[rng.permutation(len(pairs))[:n]]
    return W.Batch(np.concatenate([a.coords, b.coords]), np.concatenate([a.offsets, b.offsets + a.coords.shape[0]]),
                   np.concatenate([a.counts, b.counts]), np.ascontiguousarray(pairs), "mixed")


def _run(engine, b, bucket_kernels, null_status=False):
    import torch
    ctx = engine.Context(0)
    if bucket_kernels:  # a caller's own choice of a variant is kept at every batch size
        for kind in ("gjk", "epa"):
            for k, (lanes, blocks) in enumerate(ctx.kernel_choice()[kind]):
                ctx.set_kernel_choice(kind, k, lanes, blocks)
    pool = engine.Pool(ctx, b.counts)
    pool.upload(b.coords)
    pairs = torch.from_numpy(b.pairs).cuda()
    out = []
    fused = engine.run(ctx, pool, pairs, engine.MODE_GJK_EPA)
    out.append((fused.to_host(), ctx.work_counts(), ctx.last_launches))
    g = engine.run(ctx, pool, pairs, engine.MODE_GJK, engine.Results(b.n_pairs, pairs.device))
    out.append((g.to_host(), ctx.work_counts(), ctx.last_launches))
    e = engine.run(ctx, pool, pairs, engine.MODE_EPA, g)
    out.append((e.to_host(), ctx.work_counts(), ctx.last_launches))
    ctx.synchronize()
    return out


@pytest.mark.parametrize("n", [1, 2, 33, 500, 2048, 2049, 4096, 4097, 24576, 24577])
def test_every_route_gives_the_bucket_kernels_results(engine, n):
    b = _batch(n)
    if n > 4:
        b.pairs[2, 1] = b.n_bodies  # bad input
        b.pairs[3, 0] = -1
    ref, got = _run(engine, b, True), _run(engine, b, False)
    for (r, rw, rl), (g, gw, gl), mode in zip(ref, got, ("fused", "gjk", "epa")):
        for k in ("dist", "normal", "status"):
            assert r[k].tobytes() == g[k].tobytes(), (mode, k)
        assert r["simplex"].tobytes() == g["simplex"].tobytes(), mode
        for k in ("gjk", "epa", "polish", "refine", "refine_full", "epa_spill", "epa_late"):
            assert rw[k] == gw[k], (mode, k, rw, gw)
        assert (gl == 1) == (n <= (4096 if mode == "gjk" else 2048)), (mode, gl, rl)
