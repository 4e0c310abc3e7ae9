"""A host call that fails after the points are on their way to the device has done with the
caller's arrays when it returns: they may be unmapped at once (the device reads them in place
where it can), and the next call is none the worse."""
import ctypes
import mmap

import numpy as np
import pytest

from ogx import _lib

pytestmark = pytest.mark.gpu

POLY = {np.float32: _lib.POLYTOPE_DTYPE,
        np.float64: np.dtype([("numpoints", "<i4"), ("s", "<f8", (3,)), ("s_idx", "<i4"), ("coord", "<u8")], align=True)}


@pytest.mark.parametrize("dtype,name", [(np.float32, "ogx_compute_gjk_epa_indexed"),
                                        (np.float64, "ogx_compute_gjk_epa_indexed_f64")])
def test_arrays_may_go_after_a_bad_pair(engine, dtype, name):
    L = _lib.load()
    P, I = ctypes.c_void_p, ctypes.c_int
    fn = getattr(L, name)
    fn.restype, fn.argtypes = I, [I, I, P, P, P, P, P]
    nb, points = 4000, 500
    size = nb * points * 3 * np.dtype(dtype).itemsize
    f = np.dtype(dtype).itemsize
    smp, dist, nrm = np.zeros(nb * (184 if f == 8 else 108), np.uint8), np.zeros(nb, dtype), np.zeros((nb, 3), dtype)
    for bad in (True, False, True, False):
        m = mmap.mmap(-1, size)
        x = np.frombuffer(m, dtype)
        x[:] = np.random.default_rng(1).normal(size=x.size)
        d = np.zeros(nb, POLY[dtype])
        d["numpoints"] = points
        d["coord"] = x.ctypes.data + np.arange(nb, dtype=np.uint64) * np.uint64(points * 3 * f)
        pairs = np.stack([np.arange(nb), np.roll(np.arange(nb), 1)], 1).astype(np.int32)
        if bad:
            pairs[-1, 1] = nb
        rc = fn(nb, nb, *[P(a.ctypes.data) for a in (d, pairs, smp, dist, nrm)])
        del x
        m.close()
        assert (rc != 0) == bad, L.ogx_last_error()
    assert np.isfinite(dist).all()
