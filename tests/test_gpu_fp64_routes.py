"""The FP64 drop-in's two ways to the device -- points read where the caller keeps them, or
narrowed and gathered on the host -- give the same bits: odd sizes, arrays that are not
aligned to doubles, values that overflow or vanish as floats, non-finite coordinates; pairs
and indexed calls, the smallest batch and one with more pairs than warps on the device."""
import ctypes

import numpy as np
import pytest

from ogx import _lib

pytestmark = pytest.mark.gpu

POLY64 = np.dtype([("numpoints", "<i4"), ("s", "<f8", (3,)), ("s_idx", "<i4"), ("coord", "<u8")], align=True)
SMP64 = np.dtype([("nvrtx", "<i4"), ("vrtx", "<f8", (4, 3)), ("vrtx_idx", "<i4", (4, 2)),
                  ("witnesses", "<f8", (2, 3))], align=True)


def _bodies(nb, seed):
    g = np.random.default_rng(seed)
    counts = g.choice([1, 2, 3, 4, 5, 7, 8, 9, 31, 32, 33, 127, 130, 255, 257, 513], nb)
    off = np.concatenate([[0], np.cumsum(counts)[:-1]])
    pts = g.normal(size=(int(counts.sum()), 3))
    pts /= np.linalg.norm(pts, axis=1, keepdims=True)
    pts += np.repeat(g.uniform(-4, 4, (nb, 3)), counts, axis=0)
    return pts, counts, off


def _call(pts, counts, off, indexed, misalign=0):
    raw = np.zeros(pts.nbytes + 16, np.uint8)
    raw[misalign:misalign + pts.nbytes] = np.frombuffer(pts.tobytes(), np.uint8)
    nb = len(counts)
    d = np.zeros(nb, POLY64)
    d["numpoints"] = counts
    d["coord"] = raw.ctypes.data + misalign + 24 * off.astype(np.uint64)
    n = nb // 2
    smp, dist, nrm = np.zeros(n, SMP64), np.zeros(n), np.zeros((n, 3))
    P, I = ctypes.c_void_p, ctypes.c_int
    L = _lib.load()
    out = [P(smp.ctypes.data), P(dist.ctypes.data), P(nrm.ctypes.data)]
    if indexed:
        pairs = np.arange(2 * n, dtype=np.int32).reshape(n, 2)
        fn = L.ogx_compute_gjk_epa_indexed_f64
        fn.restype, fn.argtypes = I, [I, I, P, P, P, P, P]
        _lib.check(fn(nb, n, P(d.ctypes.data), P(pairs.ctypes.data), *out))
    else:
        a, b = np.ascontiguousarray(d[0::2]), np.ascontiguousarray(d[1::2])
        fn = L.ogx_compute_gjk_epa_f64
        fn.restype, fn.argtypes = I, [I, P, P, P, P, P]
        _lib.check(fn(n, P(a.ctypes.data), P(b.ctypes.data), *out))
    return [x.view(np.uint8).reshape(n, -1).copy() for x in (smp, dist, nrm)], dist


@pytest.mark.parametrize("indexed", [False, True])
@pytest.mark.parametrize("n", [1, 33, 3000])
def test_fp64_routes_agree(engine, monkeypatch, n, indexed):
    pts, counts, off = _bodies(2 * n, 11 + n)
    if n > 1:
        # values that a float cannot hold, and bad input, in bodies of their own
        for k, v in ((0, 1e300), (7, 1e-300), (12, np.nan), (21, np.inf)):
            pts[off[k], 1] = v
    monkeypatch.setenv("OGX_COMPAT_GATHER", "1")
    want, dist = _call(pts, counts, off, indexed)
    if n > 1:
        assert np.isnan(dist[[0, 6, 10]]).all() and np.isfinite(dist[30:]).all()
    monkeypatch.setenv("OGX_COMPAT_GATHER", "0")
    for misalign in (0, 4):
        got, _ = _call(pts, counts, off, indexed, misalign)
        for x, y in zip(got, want):
            assert np.array_equal(x, y)
