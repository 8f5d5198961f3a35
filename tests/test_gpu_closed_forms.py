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
from oracle.trajectory_oracle import trajectory
from radiacuda_b200 import _native, model

LD = np.longdouble
EPS = 2.0 ** -52


@pytest.fixture(autouse=True)
def fixed_steps(rad):
    """One Runge-Kutta step per interval, whatever a test before left set."""
    rad.FldCmpPrc("PrcCoord->-1,PrcAngle->-1")


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


def _octasphere(levels):
    """A convex polyhedron of 8 * 4^levels triangles."""
    V = [np.array(v, float) for v in ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1))]
    F = [[a, b, c] for a in (0, 1) for b in (2, 3) for c in (4, 5)]
    for _ in range(levels):
        G = []
        for a, b, c in F:
            m = []
            for i, j in ((a, b), (b, c), (c, a)):
                p = V[i] + V[j]
                p = p / np.linalg.norm(p)
                k = next((q for q, v in enumerate(V) if np.abs(v - p).max() < 1e-12), None)
                if k is None:
                    k = len(V)
                    V.append(p)
                m.append(k)
            G += [[a, m[0], m[2]], [m[0], b, m[1]], [m[2], m[1], c], m]
        F = G
    return np.array(V), F


def _poly_H(P, V, faces, M):
    """H of a convex polyhedron in long double: per face the solid angle and
    the logarithms of its edges."""
    V, P, M = (np.asarray(a, LD) for a in (V, P, M))
    cen = V.mean(0)
    H = np.zeros_like(P)
    for f in faces:
        w = V[f]
        n = np.cross(w[1] - w[0], w[2] - w[0])
        n /= np.sqrt((n * n).sum())
        if (n * (w[0] - cen)).sum() < 0:
            n, w = -n, w[::-1]
        s = (M * n).sum()
        r = w[None] - P[:, None]
        R = np.sqrt((r * r).sum(-1))
        om = np.zeros(len(P), LD)
        for j in range(1, len(f) - 1):
            i = (0, j, j + 1)
            num = (r[:, 0] * np.cross(w[j] - w[0], w[j + 1] - w[0])).sum(-1)
            d = lambda a, b: (r[:, i[a]] * r[:, i[b]]).sum(-1)
            den = R[:, 0] * R[:, j] * R[:, j + 1] + d(0, 1) * R[:, j + 1] + d(0, 2) * R[:, j] + d(1, 2) * R[:, 0]
            om -= 2 * np.arctan2(num, den)
        H += s * om[:, None] * n
        for j in range(len(f)):
            k = (j + 1) % len(f)
            e = w[k] - w[j]
            l = np.sqrt((e * e).sum())
            L = np.log1p(l * (R[:, j] + R[:, k] + l) / (R[:, j] * R[:, k] + (r[:, j] * r[:, k]).sum(-1)))
            H += s * L[:, None] * np.cross(e / l, n)
    return (H / (4 * LD(np.pi))).astype(float)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["double", "fast"])
@pytest.mark.parametrize("npts", [1, 127, 129, 700])
@pytest.mark.parametrize("ntets", [1, 2, 15, 16, 17, 33])
def test_tetrahedra(cuda, rad, ntets, npts, precision):
    """Tiles of up to 16 units and 64 faces, blocks of 128 points.  Vertices
    rebuilt from the face frames are off by a few ulp of their coordinates
    (below 8); 0.01 from a face or edge that changes a term by at most
    8 * 10 ulp / 0.01 = 2e-12."""
    rng = np.random.default_rng(ntets)
    rad.UtiDelAll()
    rad.FldLenRndSw("off")
    faces = [[1, 2, 3], [1, 4, 2], [2, 4, 3], [3, 4, 1]]
    base = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], float)
    V = [1.5 * np.array([k % 4, (k // 4) % 4, k // 16]) + base + rng.uniform(-0.1, 0.1, (4, 3)) for k in range(ntets)]
    M = rng.normal(size=(ntets, 3))
    obj = rad.ObjCnt([rad.ObjPolyhdr(v, faces, m) for v, m in zip(V, M)])
    P = rng.uniform(-1, 7, size=(npts, 3))
    exp = sum(_poly_H(P, v, [[i - 1 for i in f] for f in faces], m) for v, m in zip(V, M))
    got = rad.Fld(obj, "h", P, precision=precision)
    # the long double sums lose half their digits next to an edge too: keep to points off them
    far = np.array([min(np.abs(np.linalg.norm(p - v, axis=1)).min() for v in V) > 0.05 for p in P])
    assert np.abs(got - exp)[far].max(initial=0.0) <= 2e-12 * np.sqrt(ntets)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", ["prism", "octahedron", "sphere128"])
def test_polyhedra_by_faces(cuda, rad, shape):
    """Faces of more than three vertices, and more triangle faces than one
    staged tile holds: the general kernel.  Far points too."""
    rng = np.random.default_rng(5)
    rad.UtiDelAll()
    rad.FldLenRndSw("off")
    if shape == "prism":
        a = np.arange(5) * 2 * np.pi / 5
        V = np.concatenate([np.stack([np.cos(a), np.sin(a), np.full(5, z)], 1) for z in (-0.7, 0.9)])
        F = [[4, 3, 2, 1, 0], [5, 6, 7, 8, 9]] + [[k, (k + 1) % 5, 5 + (k + 1) % 5, 5 + k] for k in range(5)]
    else:
        V, F = _octasphere(0 if shape == "octahedron" else 2)
    M = np.array([0.4, -1.1, 0.7])
    obj = rad.ObjPolyhdr(V, [[i + 1 for i in f] for f in F], M)
    for scale in (1.5, 30.0):
        P = rng.uniform(-scale, scale, size=(300, 3))
        exp = _poly_H(P, V, F, M)
        # a few ulp of rebuilt vertices at 1e-3 or more from every edge
        assert np.abs(rad.Fld(obj, "h", P) - exp).max() <= 64 * EPS * len(F) / 1e-3 * 1e-1
    # inside, B carries the magnetization
    P = rng.uniform(-0.3, 0.3, size=(20, 3))
    assert np.abs(rad.Fld(obj, "b", P) - (_poly_H(P, V, F, M) + M)).max() <= 1e-12
    # on a face, an edge and a corner with the guards on: finite
    rad.FldLenRndSw("on")
    P = np.array([V[F[0]].mean(0), 0.5 * (V[F[0][0]] + V[F[0][1]]), V[0]])
    assert np.all(np.isfinite(rad.Fld(obj, "b", P)))
    rad.FldLenRndSw("off")


@pytest.mark.gpu
@pytest.mark.parametrize("ntets,npts", [(1, 1), (31, 130), (32, 32767), (33, 32768), (65, 33001)])
def test_tetrahedra_with_fp32_terms(cuda, rad, ntets, npts):
    """Near and far pairs, tiles of 32 tetrahedra, point sets just below and
    above the size that is put in Morton order.  A tetrahedron's terms are its 6
    edge integrals, about 2 l / R each with weights up to 1.4 |M| / (4 pi); an
    FP32 term is off by at most 4 units of 2^-24, so B by at most
    6 * 2 * 1.4 / (4 pi) * 4 * 2^-24 |M| l / R = 3.2e-7 |M| l / R a tetrahedron,
    twice that with the solid angles."""
    rng = np.random.default_rng(npts)
    rad.UtiDelAll()
    rad.FldLenRndSw("off")
    faces = [[1, 2, 3], [1, 4, 2], [2, 4, 3], [3, 4, 1]]
    base = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], float)
    V = [1.2 * np.array([k % 5, (k // 5) % 5, k // 25]) + base + rng.uniform(-0.1, 0.1, (4, 3)) for k in range(ntets)]
    M = rng.normal(size=(ntets, 3)) + [0, 0, 3.0]
    obj = rad.ObjCnt([rad.ObjPolyhdr(v, faces, m) for v, m in zip(V, M)])
    P = rng.uniform(-6, 14, size=(npts, 3))
    b64 = rad.Fld(obj, "b", P, precision="fast")
    b32 = rad.Fld(obj, "b", P, precision="single")
    R = np.array([[np.linalg.norm(p - v.mean(0)) for v in V] for p in P[:2000]])
    far = R.min(1) > 1.0
    bound = 6.4e-7 * (np.linalg.norm(M, axis=1) * 1.6 / R).sum(1)
    assert np.all((np.linalg.norm(b32 - b64, axis=1)[:2000] <= bound)[far])
    # the order of the points does not matter to a point (sums over chunks of
    # tetrahedra differ by FP64 rounding), nor do points that are not numbers
    sub = rad.Fld(obj, "b", np.ascontiguousarray(P[::7]), precision="single")
    assert np.abs(sub - b32[::7]).max() <= 1e-13 * np.abs(b32).max()
    Q = P.copy()
    Q[0] = np.nan
    assert np.array_equal(rad.Fld(obj, "b", Q, precision="single")[1:], b32[1:])
    assert np.array_equal(rad.Fld(obj, "m", P[:500], precision="single"), rad.Fld(obj, "m", P[:500]))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [4, 8, 12])
def test_fp32_terms_cancel_inside_a_mesh(cuda, rad, n):
    """A uniformly magnetized mesh of n^3 cubes of six tetrahedra: inner edges
    and faces carry no field, and their terms cancel to the bit only if every
    tetrahedron around an edge takes the same value for it, near and distant
    ones.  What is left are the errors of the surface's 18 n^2 edges of length
    1 at distances around n: each rounded to 2^-24 (2^-25 / 1.7 in the mean) of
    L = 1 / n, with weights up to 1.4 |M| / (4 pi) and |M| = 1.34, twice that
    with the distances' rounding: 4.2 * 2^-25 * 1.9 / (4 pi) * 0.58 = 1.1e-8,
    whatever n is."""
    rad.UtiDelAll()
    rad.FldLenRndSw("off")
    rng = np.random.default_rng(0)
    cube = [[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]]
    kuhn = [[0, 1, 2, 6], [0, 2, 3, 6], [0, 3, 7, 6], [0, 7, 4, 6], [0, 4, 5, 6], [0, 5, 1, 6]]
    V = np.stack([a.ravel() for a in np.meshgrid(*[np.arange(n + 1.0)] * 3, indexing="ij")], 1)
    V += rng.uniform(-0.02, 0.02, V.shape)
    tets = []
    for c in np.ndindex(n, n, n):
        at = [((c[0] + a) * (n + 1) + c[1] + b) * (n + 1) + c[2] + d for a, b, d in cube]
        tets += [rad.ObjPolyhdr(V[[at[i] for i in t]], [[1, 2, 3], [1, 4, 2], [2, 4, 3], [3, 4, 1]], [0.3, -0.7, 1.1])
                 for t in kuhn]
    obj = rad.ObjCnt(tets)
    P = rng.uniform(-4, n + 4, size=(20000, 3))
    P = np.ascontiguousarray(P[~np.all((P > -1) & (P < n + 1), axis=1)])
    d = rad.Fld(obj, "b", P, precision="single") - rad.Fld(obj, "b", P, precision="fast")
    assert np.sqrt((d * d).sum(axis=1).mean()) <= 1.1e-8


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 18, 19, 37, 74, 149])
def test_trajectories_do_not_depend_on_their_number(cuda, rad, n):
    """Clusters of 8, 4, 2 and 1 CTAs by the number of trajectories: the same
    rows bit for bit as one alone, coils (arc nodes, current blocks) included."""
    rad.UtiDelAll()
    rad.FldLenRndSw("off")
    rng = np.random.default_rng(1)
    blocks = [rad.ObjRecMag([4.0 * i - 60, 0.3, 20.0 + 0.1 * i], [3.0, 30.0, 5.0], rng.normal(size=3).tolist())
              for i in range(30)]
    yoke = rad.ObjCnt(blocks)
    rad.TrfZerPerp(yoke, [0, 0, 0], [1, 0, 0])
    rad.TrfZerPara(yoke, [0, 0, 0], [0, 0, 1])
    tet = rad.ObjPolyhdr([[70, 0, 5], [75, 1, 5], [71, 6, 5], [72, 2, 11]], [[1, 2, 3], [1, 4, 2], [2, 4, 3], [3, 4, 1]],
                         [0.2, 0.3, 0.9])
    obj = rad.ObjCnt([yoke, tet, rad.ObjRaceTrk([0.1, 0.2, 30.3], [2, 22], [60, 80], 30, 6, 15.0, "man", "z")])
    init = rng.uniform([-3, -2e-3, -3, -2e-3], [3, 2e-3, 3, 2e-3], size=(n, 4))
    batch = rad.FldPtcTrj(obj, 0.3, init, [-60, 59.5], 12)
    arrs = model.pack_sources(rad._objs, obj, tuple(rad._rand))
    for k in (0, n - 1):
        assert np.array_equal(batch[k], np.array(rad.FldPtcTrj(obj, 0.3, init[k], [-60, 59.5], 12)))
        # and the rows that the integrator makes of the oracle's field (B to 1e-10
        # of its scale, over 120 mm at 1e-3 / (T mm) of curvature)
        exp = trajectory(lambda q: O.field(arrs, q[None], 0)[0], 0.3, init[k], -60, 59.5, 12)
        assert np.abs(batch[k] - exp).max() <= 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 37])
def test_trajectory_items_two_to_a_lane(cuda, rad, n):
    """Arcs of 6,000 nodes, current blocks, cuboids with images and a
    polyhedron: more than 32 * 512 work items, so that lanes take several."""
    rad.UtiDelAll()
    rad.FldLenRndSw("off")
    rng = np.random.default_rng(2)
    coils = [rad.ObjArcCur([0.3 * k, 0.1, 25.0 + 9 * k], [3.0, 20.0], [0.2, 0.2 + 1.1 * (k + 1)], 7.0, 6000, 12.0, "man", "z")
             for k in range(3)]
    blocks = rad.ObjCnt([rad.ObjRecMag([4.0 * i - 20, 0.3, -22.0 - i], [3.0, 30.0, 5.0], rng.normal(size=3).tolist())
                         for i in range(11)])
    rad.TrfZerPara(blocks, [0, 0, 0], [0, 0, 1])
    rest = [rad.ObjRecCur([30.2, 0.4, 18.3], [4.0, 40.0, 6.0], [0.0, 9.0, 0.0]),
            rad.ObjPolyhdr([[70, 0, 5], [75, 1, 5], [71, 6, 5], [72, 2, 11]], [[1, 2, 3], [1, 4, 2], [2, 4, 3], [3, 4, 1]],
                           [0.2, 0.3, 0.9]), rad.ObjBckg([0.01, -0.02, 0.03])]
    obj = rad.ObjCnt(coils + [blocks] + rest)
    arrs = model.pack_sources(rad._objs, obj, tuple(rad._rand))
    init = rng.uniform([-3, -2e-3, -3, -2e-3], [3, 2e-3, 3, 2e-3], size=(n, 4))
    got = np.asarray(rad.FldPtcTrj(obj, 0.3, init, [-60, 59.5], 6))
    for k in (0, n - 1):
        exp = trajectory(lambda q: O.field(arrs, q[None], 0)[0], 0.3, init[k], -60, 59.5, 6)
        assert np.abs(got[k] - exp).max() <= 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("n_traj", [1, 18, 37, 74, 149])
@pytest.mark.parametrize("n_src", [1, 257, 513, 1025, 16385])
def test_cluster_exchange_with_cheap_sources(cuda, rad, n_src, n_traj):
    """Clusters of 1 to 8 CTAs on sources that cost almost nothing (uniform
    fields), so that a CTA's first sums go to its cluster's other CTAs right
    after the launch; 16,385 sources put two items on a lane.  The field is a
    sum of n_src numbers: B is off by at most n_src eps sum|b|, the angles by
    that times length / momentum, the positions by the length once more; the
    integrator's own rounding is 64 ulp of the rows."""
    rad.UtiDelAll()
    rad.FldLenRndSw("off")
    rng = np.random.default_rng(n_src)
    b = rng.uniform(0.2, 1.0, size=(n_src, 3)) * [0.3, 0.5, -0.4] / n_src
    obj = rad.ObjCnt([rad.ObjBckg(v.tolist()) for v in b])
    init = rng.uniform([-3, -2e-3, -3, -2e-3], [3, 2e-3, 3, 2e-3], size=(n_traj, 4))
    energy, lims, npts = 0.3, (-10.0, 9.5), 5
    got = np.asarray(rad.FldPtcTrj(obj, energy, init, list(lims), npts))
    B = b.sum(axis=0)
    ang = n_src * 2.0 ** -53 * np.abs(b).sum() * 2.99792458e5 / (1e9 * energy) * (lims[1] - lims[0])
    for k in (0, n_traj - 1):
        exp = trajectory(lambda P: B, energy, init[k], *lims, npts)
        bound = np.array([0.0, ang * 20.0, ang, ang * 20.0, ang]) + 64 * 2.0 ** -52 * np.abs(exp).max(axis=0)
        assert np.all(np.abs(got[k] - exp) <= bound)
    rad.FldLenRndSw("on")
