"""The sub-distance step on exact points takes over predicates that FP32 decides on the rounded
points: each of them has the sign of the exact value, also where the points' rounding is as
large as the tetrahedron (bodies far apart for their size)."""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

import far_bodies

PB_D = 7
PAIRS = [(0, 1), (1, 0), (0, 2), (2, 0), (1, 2), (2, 1)]


def step_bits(twin, n, p):
    fn = twin._lib_twin.twin_step_bits
    fn.argtypes = [ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 4
    p = np.ascontiguousarray(p, np.float32)
    out = [np.zeros(len(p), np.uint32) for _ in range(3)]
    fn(len(p), n, p.ctypes.data, *[x.ctypes.data for x in out])
    return out


def tetrahedra(g, count, apart, thickness):
    """Points a - b of 4-point steps: tetrahedra of size 1, `thickness` thick, `apart` away."""
    x = g.normal(size=(count, 4, 3))
    x[:, :, 2] *= thickness
    q, _ = np.linalg.qr(g.normal(size=(count, 3, 3)))
    x = np.einsum("nij,nkj->nki", q, x)
    b = g.normal(size=(count, 1, 3))
    d = g.normal(size=(count, 1, 3))
    d *= apart / np.linalg.norm(d, axis=2, keepdims=True)
    return np.concatenate([x + b + d, np.broadcast_to(b, x.shape)], 2).astype(np.float32)


def rational_bits(n, p):
    """The 13 predicates of one step in rational arithmetic."""
    P = [[Fraction(float(a)) - Fraction(float(b)) for a, b in zip(r[:3], r[3:])] for r in p[:n]]

    def dot(a, b):
        return sum(x * y for x, y in zip(a, b))

    def cross(a, b):
        return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]
    q = P[n - 1]
    e = [[x - y for x, y in zip(P[j], q)] for j in range(n - 1)]
    bits = 0
    for k in range(n - 1):
        bits |= (dot(q, e[k]) < 0) << k
    for k, (i, j) in enumerate(PAIRS):
        if max(i, j) < n - 1:
            bits |= (dot(q, cross(e[i], cross(e[i], e[j]))) < 0) << (PB_D + k)
    if n == 4:
        bits |= (dot(e[1], cross(e[0], e[2])) <= 0) << 3
        for k, (i, j) in ((4, (1, 0)), (5, (0, 2)), (6, (2, 1))):
            bits |= (dot(q, cross(P[i], P[j])) <= 0) << k
    return bits


MASK = {2: 0x1, 3: 0x3 | 0x3 << PB_D, 4: 0x1fff}


@pytest.mark.parametrize("n", [2, 3, 4])
@pytest.mark.parametrize("apart", [0.1, 1, 10, 100, 1e3, 1e4, 1e6])
def test_known_bits_have_the_exact_sign(twin, n, apart):
    g = np.random.default_rng(int(7 * apart) + n)
    for thickness in (1, 1e-2, 1e-4, 1e-6, 0):
        p = tetrahedra(g, 20000, apart, thickness)
        bits, known, exact = step_bits(twin, n, p)
        wrong = (bits ^ exact) & known & MASK[n]
        # (FP64 is exact enough to be the judge except next to zero: those are looked at again)
        for i in np.nonzero(wrong)[0]:
            assert ((int(bits[i]) ^ rational_bits(n, p[i])) & int(known[i]) & MASK[n]) == 0, (thickness, p[i])
    if apart <= 1:  # and they are what most steps decide on
        p = tetrahedra(g, 20000, apart, 1)
        bits, known, _ = step_bits(twin, n, p)
        assert (((known & MASK[n]) == MASK[n]).mean()) > 0.5


@pytest.mark.parametrize("n", [2, 3, 4])
@pytest.mark.parametrize("scale", [-140, -60, -45, -38, -30, -25, -20, 20, 28, 31, 33, 40, 63, 100, 126])
def test_known_bits_at_every_scale(twin, n, scale):
    """Up to where products of four lengths overflow, and down to where they vanish."""
    g = np.random.default_rng(abs(scale) + n)
    for thickness in (1, 1e-3, 0):
        p = tetrahedra(g, 4000, 1, thickness).astype(np.float64) * 2.0 ** scale
        p *= 2.0 ** g.integers(-12, 1, (len(p), 4, 1))  # points of different sizes
        p = np.clip(p, -3e38, 3e38).astype(np.float32)
        bits, known, exact = step_bits(twin, n, p)
        for i in np.nonzero((bits ^ exact) & known & MASK[n])[0]:
            assert ((int(bits[i]) ^ rational_bits(n, p[i])) & int(known[i]) & MASK[n]) == 0, (thickness, p[i])
    # (sizes 2^-12 to 1 times the scale: all of them out of range at the ends, some in it between)
    any_known = ((known & MASK[n]) != 0).any()
    assert any_known if -20 <= scale <= 28 else True
    assert not any_known if scale <= -45 or scale >= 63 else True


@pytest.mark.parametrize("exponent", [31, 50])
@pytest.mark.parametrize("apart", [3, 30])
def test_large_bodies_whose_products_overflow(orc, twin, apart, exponent):
    b = far_bodies.batch(5 + apart, 3000, apart, 0.0, "line")
    b.coords *= np.float32(2.0 ** exponent)
    o = orc.run(b.coords, b.offsets, b.counts, b.pairs, mode=orc.MODE_GJK, precision="f64", threads=8)
    r = twin.run(b, mode=1)
    assert (np.abs(r["dist"] - o["dist"]) <= 1e-5 * o["dist"]).all()


def test_fp64_bits_are_the_rational_ones(twin):
    g = np.random.default_rng(3)
    for n in (2, 3, 4):
        p = tetrahedra(g, 200, 3, 0.1)
        _, _, exact = step_bits(twin, n, p)
        assert [int(x) & MASK[n] for x in exact] == [rational_bits(n, r) for r in p]


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("kind,thickness", [("disk", 0.0), ("disk", 1e-5), ("disk", 1e-3), ("dome", 1e-5),
                                            ("dome", 1e-3), ("line", 1e-5), ("ball", 1.0)])
@pytest.mark.parametrize("apart", [3, 10, 100, 1e3, 1e4])
def test_bodies_far_apart_for_their_size(orc, twin, apart, kind, thickness, mode):
    for size2 in (1.0, 1e-3):
        b = far_bodies.batch(int(apart) + 7, 4000, apart, thickness, kind, size2)
        o = orc.run(b.coords, b.offsets, b.counts, b.pairs, mode=orc.MODE_GJK_EPA, precision="f64", threads=8)
        r = twin.run(b, mode=mode)
        if mode == 1:
            r["normal"] = None
        bad = far_bodies.errors(b, r, o)
        assert len(bad) == 0, (size2, bad[:5], r["dist"][bad[:5]], o["dist"][bad[:5]])


def test_projection_on_a_triangle_keeps_its_signs(twin):
    """The normal of the plane is that of (newest, second, first): where it has a zero component, the
    zero's sign is part of the result."""
    fn = twin._lib_twin.twin_triangle_step
    fn.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 3
    g = np.random.default_rng(9)
    p = g.integers(-4, 5, (4000, 3, 3)).astype(np.float64)
    p[:, :, 2] = g.integers(1, 3, (4000, 1))  # in a plane z = const: the origin projects on (0, 0, z)
    left, v = np.zeros(len(p), np.int32), np.zeros((len(p), 3))
    fn(len(p), p.ctypes.data, left.ctypes.data, v.ctypes.data)
    on = left == 3
    assert on.sum() > 100
    q1, q2, q3 = p[on, 2], p[on, 1], p[on, 0]
    a, b = q1 - q2, q1 - q3
    n = np.stack([a[:, 1] * b[:, 2] - a[:, 2] * b[:, 1], a[:, 2] * b[:, 0] - a[:, 0] * b[:, 2],
                  a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]], 1)
    d = (n[:, 0] * q1[:, 0] + n[:, 1] * q1[:, 1]) + n[:, 2] * q1[:, 2]
    with np.errstate(invalid="ignore"):
        want = n * (d / ((n[:, 0] * n[:, 0] + n[:, 1] * n[:, 1]) + n[:, 2] * n[:, 2]))[:, None]
    assert v[on].tobytes() == want.tobytes()
