"""The FP64 drop-in on bodies of every odd size against the FP64 oracle on the same doubles, with
the points read by the device where the caller keeps them and gathered on the host."""
import ctypes

import numpy as np
import pytest

import parity
from test_gpu_fp64_routes import _bodies, _call

pytestmark = pytest.mark.gpu


def _device_reads_pageable():
    cu = ctypes.CDLL("libcuda.so.1")
    v = [ctypes.c_int(0), ctypes.c_int(0)]
    for x, attr in zip(v, (88, 100)):  # pageable access, and through the host's page tables
        assert cu.cuDeviceGetAttribute(ctypes.byref(x), attr, 0) == 0
    return all(x.value for x in v)


@pytest.mark.parametrize("gather", ["1", "0"])
@pytest.mark.parametrize("indexed", [False, True])
def test_odd_sizes_against_the_oracle(engine, orc, monkeypatch, indexed, gather):
    if gather == "0" and not _device_reads_pageable():
        pytest.skip("the device does not read pageable host memory")
    pts, counts, off = _bodies(4000, 23)
    monkeypatch.setenv("OGX_COMPAT_GATHER", gather)
    _, dist = _call(pts, counts, off, indexed)
    pairs = np.arange(4000, dtype=np.int32).reshape(-1, 2)
    o = orc.run(pts, off, counts, pairs, mode=orc.MODE_GJK, precision="f64", threads=8)
    sep = o["dist"] > parity.BAND * 8  # (coordinates up to 5)
    assert sep.sum() > 1000
    assert (np.abs(dist[sep] - o["dist"][sep]) <= parity.REL * o["dist"][sep]).all()
