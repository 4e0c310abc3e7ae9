"""World points of the serving loop's transform: the FP32 route gives the FP64 evaluation's
float for every input that it settles, and leaves the others to FP64."""
import ctypes

import numpy as np
import pytest

import twin_bind

N = 200_000


def _world(xf, p):
    fn = twin_bind._lib_twin.twin_world_points
    fn.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 4
    xf, p = np.ascontiguousarray(xf, np.float32), np.ascontiguousarray(p, np.float32)
    out, ok = np.empty_like(p), np.empty(len(p), np.uint8)
    fn(len(p), xf.ctypes.data, p.ctypes.data, out.ctypes.data, ok.ctypes.data)
    return out, ok.astype(bool)


def _exact(xf, p):
    x, q = np.asarray(xf, np.float32).astype(np.float64), np.asarray(p, np.float32).astype(np.float64)
    with np.errstate(all="ignore"):
        w = [((x[:, 3 * k] * q[:, 0] + x[:, 3 * k + 1] * q[:, 1]) + x[:, 3 * k + 2] * q[:, 2]) + x[:, 9 + k]
             for k in range(3)]
        return np.stack(w, 1).astype(np.float32)


def _case(kind):
    g = np.random.default_rng(5)
    q, _ = np.linalg.qr(g.normal(size=(N, 3, 3)))
    t = g.uniform(-50, 50, (N, 3))
    p = g.normal(size=(N, 3))
    if kind == "cancel":  # the translation takes the rotated point away, to the last bits
        t = -np.einsum("nij,nj->ni", q.astype(np.float32).astype(np.float64), p.astype(np.float32))
    elif kind == "ties":  # sums half way between two floats, and next to it
        q = np.broadcast_to(np.eye(3), q.shape).copy()
        p = np.ldexp(1.0 + g.integers(0, 1 << 23, (N, 3)) / (1 << 23), g.integers(-3, 4, (N, 1)))
        t = np.ldexp(np.spacing(p.astype(np.float32)).astype(np.float64), -1) * g.choice([-3, -1, -0.5, 1, 1.5, 3], (N, 3))
        t = t * (1 + g.choice([0, 2.0 ** -23, -2.0 ** -23], (N, 3)))
    elif kind == "scales":  # from below the smallest normal product to overflow
        q = q * np.ldexp(1.0, g.integers(-70, 70, (N, 1, 1)))
        p = p * np.ldexp(1.0, g.integers(-70, 70, (N, 1)))
        t = t * np.ldexp(1.0, g.integers(-149, 120, (N, 3)))
    elif kind == "special":
        v = np.array([0.0, -0.0, 1.0, -1.0, 2.0 ** -149, 2.0 ** -126, 3e38, -3e38, np.inf, -np.inf, np.nan, 0.1])
        q, p, t = (v[g.integers(0, len(v), s)] for s in (q.shape, p.shape, t.shape))
    return np.concatenate([q.reshape(N, 9), t], 1), p


@pytest.mark.parametrize("kind", ["poses", "cancel", "ties", "scales", "special"])
def test_world_points_are_the_fp64_evaluation(kind):
    xf, p = _case(kind)
    got, settled = _world(xf, p)
    want = _exact(xf, p)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got.view(np.int32)[~nan], want.view(np.int32)[~nan])  # bits: -0.0 too
    if kind == "poses":
        assert settled.mean() > 0.99
    if kind == "ties":
        assert not settled.all()
