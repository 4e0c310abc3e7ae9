"""Exact supports: the first point of a body with the largest FP64 value along a direction, at
every scale (to where FP32 products overflow), with ties and near ties."""
import ctypes

import numpy as np
import pytest

from ogx import pool as P


@pytest.mark.parametrize("kind", ["random", "ties", "near"])
@pytest.mark.parametrize("scale", [-60, -20, 0, 20, 60, 63, 68, 74, 90, 120])
def test_exact_support(twin, scale, kind):
    fn = twin._lib_twin.twin_exact_support
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 3
    g = np.random.default_rng(scale + 200)
    for n in (1, 2, 3, 5, 8, 33, 200):
        x = g.normal(size=(n, 3))
        if kind == "ties":
            x = np.round(x)
        elif kind == "near":
            x = x[:1] + x * 2.0 ** -22
        x = np.clip(x * 2.0 ** scale, -3e38, 3e38).astype(np.float32)
        d = g.normal(size=(300, 3)) * 2.0 ** np.minimum(scale, 100)
        pool, quad = P.pack(x, np.array([n], np.int32))
        assert quad[0] == 0
        idx, val = np.zeros(len(d), np.int32), np.zeros(len(d))
        fn(pool.ctypes.data, n, len(d), d.ctypes.data, idx.ctypes.data, val.ctypes.data)
        p = x.astype(np.float64)
        v = (p[None, :, 0] * d[:, :1] + p[None, :, 1] * d[:, 1:2]) + p[None, :, 2] * d[:, 2:]
        assert np.array_equal(idx, v.argmax(1)), n
        assert np.array_equal(val, v.max(1)), n
