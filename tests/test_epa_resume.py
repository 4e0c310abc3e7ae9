"""A contact that outgrows EPA's small capacity is either continued at full capacity from where
it stopped or started again there: the same result, with FP32 face planes and with FP64 ones
(the one-warp-per-pair route starts again, the bucket kernels continue what they saved)."""
import functools

import pytest

from ogx import _lib, workloads as W

ESCALATE, POLISH, PLANES64 = 1, 2, 8


@functools.lru_cache(maxsize=1)
def _batch():
    return W.ellipsoid(seed=19, n_pairs=600, lo=1500, hi=6000)


@pytest.mark.parametrize("flags", [0, ESCALATE, ESCALATE | POLISH, PLANES64, ESCALATE | PLANES64,
                                   ESCALATE | POLISH | PLANES64])
@pytest.mark.parametrize("cap", [25, 26, 64])
def test_continued_expansions_are_the_restarted_ones(twin, flags, cap):
    b = _batch()
    c = twin.config(flags=flags, epa_max_iter=cap)
    want, got = twin.run(b, mode=2, cfg=c), twin.run(b, mode=3, cfg=c)
    if cap == 64:
        assert (want["iters"][:, 1] > 24).sum() > 20  # expansions that outgrow the small capacity
    for k in ("dist", "normal", "status", "iters", "simplex"):
        assert want[k].tobytes() == got[k].tobytes(), k


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [ESCALATE | POLISH, ESCALATE | POLISH | PLANES64, PLANES64])
def test_routes_agree_on_large_expansions(engine, flags):
    import torch
    b = _batch()
    cfg = _lib.default_config()
    cfg.flags = flags
    out = []
    for bucket_kernels in (False, True):
        ctx = engine.Context(0, cfg)
        if bucket_kernels:
            for kind in ("gjk", "epa"):
                for k, (lanes, blocks) in enumerate(ctx.kernel_choice()[kind]):
                    ctx.set_kernel_choice(kind, k, lanes, blocks)
        pool = engine.Pool(ctx, b.counts)
        pool.upload(b.coords)
        r = engine.run(ctx, pool, torch.from_numpy(b.pairs).cuda(), engine.MODE_GJK_EPA)
        ctx.synchronize()
        assert ctx.work_counts()["epa_spill"] > 20
        out.append(r.to_host())
    for k in ("dist", "normal", "status", "simplex"):
        assert out[0][k].tobytes() == out[1][k].tobytes(), k


@pytest.mark.gpu
def test_both_routes_continue_large_expansions(engine):
    import torch
    b = _batch()
    for bucket_kernels in (False, True):
        ctx = engine.Context(0)
        if bucket_kernels:
            for k, (lanes, blocks) in enumerate(ctx.kernel_choice()["epa"]):
                ctx.set_kernel_choice("epa", k, lanes, blocks)
        pool = engine.Pool(ctx, b.counts)
        pool.upload(b.coords)
        engine.run(ctx, pool, torch.from_numpy(b.pairs).cuda(), engine.MODE_GJK_EPA)
        ctx.synchronize()
        assert (ctx.last_launches > 1) == bucket_kernels
        assert ctx.work_counts()["epa_resumed"] > 20
