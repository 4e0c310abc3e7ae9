"""Finite bodies so large that products of their coordinates overflow (from about 1e13 on):
no result is promised in contact, but every index that is read with, or returned, is one of
the bodies'.  In a process of its own, since reading out of range may end it."""
import subprocess
import sys

import pytest

CODE = """
import sys
sys.path[:0] = {path!r}
import numpy as np
import twin_bind
from ogx import workloads as W
for gen in (W.stress, W.ellipsoid, W.plain):
    b = gen(seed=3, n_pairs=600)
    b.coords = np.clip(b.coords.astype(np.float64) * 2.0 ** {scale}, -3.4e38, 3.4e38).astype(np.float32)
    for flags in (0, 3, 11):
        r = twin_bind.run(b, mode=3, cfg=twin_bind.config(flags=flags), threads=1)
        s = r["simplex"]
        assert ((s["nvrtx"] >= 1) & (s["nvrtx"] <= 4)).all()
        n = b.counts[b.pairs][:, None, :]
        assert ((s["vrtx_idx"] >= 0) & (s["vrtx_idx"] < n)).all()
"""


@pytest.mark.parametrize("scale", [30, 50, 60, 63, 66, 80, 126])
def test_indices_stay_in_range(twin, scale):
    code = CODE.format(path=sys.path, scale=scale)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-500:]
