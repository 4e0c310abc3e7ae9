"""Pairs of flat and thin bodies that lie far apart for their size, and the rules that their
results have to meet.  The rounding of the points themselves (half an ulp of a coordinate)
is then as large as the bodies' thickness, or as the bodies."""
import numpy as np

import parity
from ogx import workloads as W


def batch(seed, n_pairs, apart, thickness, kind="disk", size2=1.0):
    """n_pairs pairs of bodies of 3 to 12 points and radius 1 (the second: size2), their
    centres `apart` radii from one another in a random direction, their axes along it but for a
    tilt of 1e-6 to 1: "disk" random points of a disk, `thickness` thick; "dome" a disk bent
    outwards by `thickness`; "line" points of a segment; "ball" points of a sphere."""
    g = np.random.default_rng(seed)
    nb = 2 * n_pairs
    counts = g.integers(3, 13, nb).astype(np.int32)
    off = np.concatenate([[0], np.cumsum(counts)[:-1]])
    total = int(counts.sum())
    body = np.repeat(np.arange(nb), counts)
    r, phi = np.sqrt(g.uniform(0.05, 1, total)), g.uniform(0, 2 * np.pi, total)
    p = np.stack([r * np.cos(phi), r * np.sin(phi), thickness * g.uniform(-1, 1, total)], 1)
    if kind == "dome":
        p[:, 2] = -thickness * r * r * np.where(body % 2, -1.0, 1.0)
    elif kind == "line":
        p[:, 1:] *= thickness
    elif kind == "ball":
        p = g.normal(size=(total, 3))
        p /= np.linalg.norm(p, axis=1, keepdims=True)
    d = g.normal(size=(n_pairs, 3))
    d *= apart / np.linalg.norm(d, axis=1, keepdims=True)
    axis = np.repeat(d / apart, 2, axis=0) + g.normal(size=(nb, 3)) * 10.0 ** g.uniform(-6, 0, (nb, 1))
    q, _ = np.linalg.qr(np.concatenate([axis[:, :, None], g.normal(size=(nb, 3, 2))], 2))
    q = q[:, :, [1, 2, 0]] * np.sign(np.einsum("ni,ni->n", q[:, :, 0], axis))[:, None, None]  # z = the axis
    p = np.einsum("nij,nj->ni", q[body], p) * np.where(body % 2, size2, 1.0)[:, None]
    centre = np.zeros((nb, 3))
    centre[1::2] = d
    centre += np.repeat(g.normal(size=(n_pairs, 3)), 2, axis=0)
    pairs = np.arange(nb, dtype=np.int32).reshape(-1, 2)
    return W.Batch((p + centre[body]).astype(np.float32), off.astype(np.int64), counts, pairs, kind)


def errors(b, res, o):
    """Pairs that break a rule of tests/parity.py for separated pairs (all of them are): the
    verdict, the distance, and the bodies' separation along the normal (where there is one)."""
    d, d64 = res["dist"].astype(np.float64), o["dist"]
    assert (d64 > 0).all()
    bad = ~(d > 0) | (res["simplex"]["nvrtx"] > 3)
    bad |= ~(np.abs(d - d64) <= parity.REL * d64)
    if res.get("normal") is not None:
        n = res["normal"].astype(np.float64)
        body = np.repeat(np.arange(b.n_bodies), b.counts)
        x = b.coords.astype(np.float64)
        along = np.einsum("ij,ij->i", x, n[body // 2])  # body i belongs to pair i // 2
        gap = np.minimum.reduceat(along, b.offsets)[1::2] - np.maximum.reduceat(along, b.offsets)[0::2]
        tol = parity.EQUIV * np.maximum(parity.pair_scale(b), d64)
        bad |= ~(np.abs(np.linalg.norm(n, axis=1) - 1) <= 1e-6) | ~(gap >= d64 * (1 - parity.REL) - tol)
    return np.nonzero(bad)[0]
