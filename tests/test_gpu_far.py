"""Flat and thin bodies far apart for their size, on both routes of a call (one warp per pair,
bucket kernels): separated, at the FP64 oracle's distance, along a separating normal."""
import numpy as np
import pytest

import far_bodies

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1500, 6000])
@pytest.mark.parametrize("kind,thickness", [("disk", 0.0), ("disk", 1e-5), ("dome", 1e-3), ("line", 1e-5)])
@pytest.mark.parametrize("apart", [3, 30, 1e3, 1e4])
def test_bodies_far_apart_for_their_size(engine, orc, apart, kind, thickness, n):
    for size2 in (1.0, 1e-3):
        b = far_bodies.batch(int(apart) + n, n, apart, thickness, kind, size2)
        o = orc.run(b.coords, b.offsets, b.counts, b.pairs, mode=orc.MODE_GJK_EPA, precision="f64", threads=8)
        for mode in (engine.MODE_GJK, engine.MODE_GJK_EPA):
            r = engine.query(b, mode)
            if mode == engine.MODE_GJK:
                r["normal"] = None
            bad = far_bodies.errors(b, r, o)
            assert len(bad) == 0, (mode, size2, bad[:5], r["dist"][bad[:5]], o["dist"][bad[:5]])


@pytest.mark.parametrize("exponent", [31, 50])
def test_large_bodies_whose_products_overflow(engine, orc, exponent):
    for n in (3000, 6000):
        b = far_bodies.batch(n, n, 3, 0.0, "line")
        b.coords *= np.float32(2.0 ** exponent)
        o = orc.run(b.coords, b.offsets, b.counts, b.pairs, mode=orc.MODE_GJK, precision="f64", threads=8)
        r = engine.query(b, engine.MODE_GJK)
        assert (np.abs(r["dist"] - o["dist"]) <= 1e-5 * o["dist"]).all()
