"""The cuboid's closed form at the places where its branches change, against
extended precision.

H of a cuboid with unit magnetization is a column of its tensor, whose entries
are at most 1 in magnitude outside edges: corner sums of arctan(YZ / (XR)) and
asinh(Z / sqrt(X^2 + Y^2)) in numpy's long double.  The device form rounds a
few hundred operations, of which those on values of order one number about
thirty per entry: 8 ulp of the larger of 1 and the entry.  The offsets of a
point from the faces are rounded once in FP64 before either form uses them,
so the reference takes the rounded ones.
"""
import numpy as np
import pytest

import oracle.oracle as O
from radiacuda_b200 import _native, model

LD = np.longdouble
EPS = 2.0 ** -52


def _tensor(q, d):
    """[n, 3, 3] in long double; q = point - centre, d the full widths."""
    h = LD(0.5) * np.asarray(d, LD)
    lo, hi = (-q - 0.5 * np.asarray(d)).astype(LD), (-q + 0.5 * np.asarray(d)).astype(LD)
    T = np.zeros((len(q), 3, 3), LD)
    del h
    for i in range(8):
        s = [(i >> a) & 1 for a in range(3)]
        p = LD((-1) ** (sum(s) + 1))
        X, Y, Z = ((hi if s[a] else lo)[:, a] for a in range(3))
        R = np.sqrt(X * X + Y * Y + Z * Z)
        c = (X, Y, Z)
        for a in range(3):
            b, e = (a + 1) % 3, (a + 2) % 3
            T[:, a, a] -= p * np.arctan(c[b] * c[e] / (c[a] * R))
            L = p * np.arcsinh(c[e] / np.sqrt(c[a] ** 2 + c[b] ** 2))
            T[:, a, b] += L
            T[:, b, a] += L
    return T / (4 * LD(np.pi) + LD(1.2246467991473532e-16) * 4)


def _points(kind, d, rng):
    h = 0.5 * np.asarray(d)
    n = 400
    if kind == "around":      # every slab combination, inside too
        return rng.uniform(-3, 3, size=(n, 3)) * h
    if kind == "inside":
        return rng.uniform(-1, 1, size=(n, 3)) * h
    if kind == "far":
        return rng.uniform(-60, 60, size=(n, 3)) * h.max()
    if kind == "face":        # close to one face plane, both sides, over and beside the face
        q = rng.uniform(-1.5, 1.5, size=(n, 3)) * h
        a = rng.integers(0, 3, n)
        off = rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-9, -1, n)
        q[np.arange(n), a] = rng.choice([-1.0, 1.0], n) * h[a] * (1.0 + off)
        return q
    q = np.zeros((n, 3))      # "axis": on the symmetry axes and planes through the centre
    q[:, 0] = rng.uniform(-4, 4, n) * h[0]
    q[n // 2:, 1] = rng.uniform(-4, 4, n - n // 2) * h[1]
    return q


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1.0, 1e-13, 1e13])
@pytest.mark.parametrize("kind", ["around", "inside", "far", "face", "axis"])
@pytest.mark.parametrize("dims", [(10.0, 7.0, 4.0), (100.0, 0.3, 5.0), (2.0, 2.0, 2.0)])
def test_cuboid_tensor(cuda, rad, dims, kind, scale):
    rad.UtiDelAll()
    rad.FldLenRndSw("off")
    rng = np.random.default_rng(3)
    d = np.asarray(dims) * scale
    q = np.ascontiguousarray(_points(kind, d, rng))
    keep = np.all(np.abs(np.abs(q) - 0.5 * d) > 0, axis=1)
    q = q[keep]
    exp = _tensor(q, d)
    got = np.zeros((len(q), 3, 3))
    for b in range(3):
        h = rad.ObjRecMag([0, 0, 0], d.tolist(), np.eye(3)[b].tolist())
        got[:, :, b] = _native.field(model.pack_sources(rad._objs, h, tuple(rad._rand)), q, 1)
    bound = 8 * EPS * np.maximum(1.0, np.abs(exp).astype(float))
    assert np.all(np.abs(got - exp.astype(float)) <= bound)


@pytest.mark.gpu
def test_cuboid_guards_and_singular_points(cuda, rad):
    """Guards on: points on faces, edges and corners as the oracle has them.
    Guards off: a point on a face plane keeps an undefined normal entry."""
    d = np.array([4.0, 6.0, 8.0])
    P = np.array([[2.0, 0.3, 0.4], [2.0, 3.0, 0.4], [2.0, 3.0, 9.0], [2.0, 3.0, -4.0], [-2.0, -3.0, -4.0],
                  [2.0, 9.0, 1.0], [0.1, 3.0, 4.0 + 1e-10]])
    rad.UtiDelAll()
    for onoff in ("on", "off"):
        rad.FldLenRndSw(onoff)
        h = rad.ObjRecMag([0, 0, 0], d.tolist(), [0.3, -0.7, 1.1])
        g = model.pack_sources(rad._objs, h, tuple(rad._rand))
        for what in (0, 1):
            got, exp = _native.field(g, P, what), O.field(g, P, what)
            if onoff == "on":
                assert np.all(np.isfinite(got))
                # the reference's sums z + D with z < 0 lose up to half of the digits on an edge line's extension
                assert np.abs(got - exp).max() <= 1e-6 * np.abs(exp).max()
            else:
                assert np.array_equal(np.isfinite(got[:6]), np.isfinite(exp[:6]))
    rad.FldLenRndSw("off")
