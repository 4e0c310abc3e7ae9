"""FP64 values compared as integers by the exact supports: the ordered key of a double, over
every exponent, the special values and random bit patterns."""
import ctypes

import numpy as np

import twin_bind

L = twin_bind._lib_twin


def _doubles():
    g = np.random.default_rng(2)
    u = np.uint64
    edge = (np.arange(2048, dtype=u)[:, None] << u(52)) | np.array([0, 1, 2, (1 << 52) - 2, (1 << 52) - 1], u)
    edge = np.concatenate([edge.ravel(), edge.ravel() | (u(1) << u(63))]).view(np.float64)
    near = [0.0, -0.0, 1.0, np.nextafter(1.0, 2.0), -1.0, np.inf, -np.inf]
    return np.concatenate([np.frombuffer(g.bytes(8 << 18), np.float64), edge, near])


def test_order_key_orders_as_the_doubles_do():
    x = _doubles()
    key, back = np.empty(len(x), np.int64), np.empty(len(x))
    L.twin_order_key64(ctypes.c_int64(len(x)), *[ctypes.c_void_p(a.ctypes.data) for a in (x, key, back)])
    nan = np.isnan(x)
    assert (key[nan] == np.iinfo(np.int64).min).all()
    assert np.array_equal(back[~nan], x[~nan])
    v, k = x[~nan], key[~nan]
    o = np.argsort(v, kind="stable")
    v, k = v[o], k[o]
    assert np.array_equal(v[1:] == v[:-1], k[1:] == k[:-1]) and (k[1:] >= k[:-1]).all()
    assert k[0] > np.iinfo(np.int64).min
