"""A pose update is checked block by block (1024 entries): a NaN or an infinity of either sign
is found in the first and last entry of a block and in the ragged last block, and named by its
body; the largest finite values, zeros of either sign and subnormals pass."""
import numpy as np
import pytest

from ogx import _lib
from ogx import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_bodies", [85, 86, 257])  # 1,020, 1,032 and 3,084 entries
def test_every_place_is_checked(n_bodies):
    from ogx import serving
    scene = W.serving_scene(seed=5, n_bodies=n_bodies)
    xf = np.ascontiguousarray(scene.transforms(1), dtype=np.float32)
    n = xf.size
    bad_bits = [0x7f800000, 0xff800000, 0x7fc00000, 0xffffffff, 0x7f800001]
    with serving.Server(scene.counts, scene.local, warm_start=False) as srv:
        for i in sorted({0, 1, 1023, 1024, 2047, 2048, n - 2, n - 1} & set(range(n))):
            for u in bad_bits:
                x = xf.copy()
                x.reshape(-1).view(np.uint32)[i] = u
                with pytest.raises(_lib.OgxError) as ei:
                    srv.set_transforms(x)
                assert ei.value.status == -1 and f"body {i // 12} " in str(ei.value)
        x = np.zeros_like(xf)
        x.reshape(-1).view(np.uint32)[:6] = [0x7f7fffff, 0xff7fffff, 0x80000000, 1, 0x807fffff, 0x00800000]
        srv.set_transforms(x)
