"""Fields of bodies and at points where a closed form degenerates: collapsed
faces, negative widths, points on faces, edges and corners, extreme lengths.
The CPU oracle (the reference's formulas term by term) says what holds there.
"""
import ctypes as C

import numpy as np
import pytest

import oracle.oracle as O
from oracle.trajectory_oracle import trajectory
from radiacuda_b200 import _native, model
from test_zz_no_alloc import _device_geom

EPS = 2.0 ** -52


@pytest.fixture(autouse=True)
def fixed_steps(rad):
    """One Runge-Kutta step per interval, whatever a test before left set."""
    rad.FldCmpPrc("PrcCoord->-1,PrcAngle->-1")


def _noalloc(cuda, arrs, P, what):
    import torch

    L = _native.lib()
    L.radb200_field_noalloc.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_int, C.c_void_p]
    g, keep = _device_geom(arrs, torch, cuda)
    d_pts = torch.from_numpy(np.ascontiguousarray(P)).to(cuda)
    d_out = torch.full(P.shape, float("nan"), dtype=torch.float64, device=cuda)
    _native.check(L.radb200_field_noalloc(C.cast(C.byref(g), C.c_void_p), C.c_void_p(d_pts.data_ptr()), P.shape[0], what,
                                          C.c_void_p(d_out.data_ptr())), "radb200_field_noalloc")
    return d_out.cpu().numpy()


def _arrays(rad, obj):
    return model.pack_sources(rad._objs, obj, tuple(rad._rand))


@pytest.fixture(params=["on", "off"])
def guards(request, rad):
    rad.UtiDelAll()
    rad.FldLenRndSw(request.param)
    yield request.param
    rad.FldLenRndSw("on")


PRISM = np.array([[0, 0, 0], [1, 0, 0], [0.3, 1, 0], [0.2, 0.1, 1.1], [1.2, 0.1, 1.1], [0.5, 1.1, 1.1]])
SIDES = [[1, 2, 5, 4], [2, 3, 6, 5], [3, 1, 4, 6]]


@pytest.mark.gpu
@pytest.mark.parametrize("ends", [([1, 3, 2], [4, 5, 6]), ([1, 3, 3, 2], [4, 5, 6, 6]), ([1, 3, 3, 3, 2], [4, 5, 5, 6]),
                                  ([1, 3, 2, 2], [4, 5, 6, 6, 6]), ([1, 3, 2, 1], [4, 5, 6, 4])])
def test_collapsed_faces(cuda, rad, guards, ends):
    """A wedge written as a collapsed hexahedron: a face that names a vertex
    twice is the face that names it once, in every caller of the face form.
    The vertices' own rounding (8 ulp) at 0.05 or more from an edge changes H by
    at most 8 eps / 0.05 per edge, of 9 edges twice: 6e-13."""
    plain = rad.ObjPolyhdr(PRISM, [[1, 3, 2], [4, 5, 6]] + SIDES, [0.4, -0.6, 0.9])
    obj = rad.ObjPolyhdr(PRISM, list(ends) + SIDES, [0.4, -0.6, 0.9])
    rng = np.random.default_rng(2)
    P = np.concatenate([rng.uniform(-2, 3, size=(40, 3)), PRISM.mean(0) + rng.uniform(-0.05, 0.05, size=(5, 3))])
    P = P[[min(np.linalg.norm(np.outer(t, PRISM[j] - PRISM[i]) + PRISM[i] - p, axis=1).min()
               for t in [np.linspace(0, 1, 200)] for f in [[0, 2, 1], [3, 4, 5]] + [[v - 1 for v in s] for s in SIDES]
               for i, j in zip(f, f[1:] + f[:1])) > 0.05 for p in P]]
    a, b = _arrays(rad, plain), _arrays(rad, obj)
    for what in (0, 1, 2):
        got = _native.field(b, P, what)
        assert np.abs(got - _native.field(a, P, what)).max() <= 6e-13
        # the reference's terms lose up to four digits next to near-vertical edges
        assert np.abs(got - O.field(b, P, what)).max() <= 1e-11
        assert np.abs(_noalloc(cuda, b, P, what) - got).max() <= 6e-13
    p1, p2 = np.array([-3.0, 0.4, 2.0]), np.array([4.0, 0.7, -1.5])
    assert np.abs(np.array(_native.field_int(b, p1, p2, False, 3)[0]) -
                  np.array(_native.field_int(a, p1, p2, False, 3)[0])).max() <= 1e-11
    init = np.array([0.4, 1e-3, 1.9, -1e-3])
    row = np.array(rad.FldPtcTrj(obj, 0.05, init, [-5, 5.3], 7))
    exp = trajectory(lambda q: O.field(b, q[None], 0)[0], 0.05, init, -5, 5.3, 7)
    assert np.abs(row - exp).max() <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("ends", [([1, 3, 3, 2], [4, 5, 6, 6]), ([1, 3, 2, 1], [4, 5, 5, 6])])
def test_collapsed_faces_by_vertices_and_edges(cuda, rad, guards, ends):
    """The vertex/edge form of the same wedge: its terms are the plain one's, so
    FP64 agrees to rounding and FP32 terms to 8 units of 2^-24 of terms of
    order |M|; the interaction assembled in that form too."""
    mat = rad.MatLin([3.0, 3.0], [0.0, 0.0, 0.7])
    plain, obj = (rad.ObjPolyhdr(PRISM, e + SIDES, [0.4, -0.6, 0.9]) for e in ([[1, 3, 2], [4, 5, 6]], list(ends)))
    P = np.random.default_rng(6).uniform(1.5, 4, size=(50, 3))
    for precision, tol in (("fast", 1e-14), ("single", 8 * 2.0 ** -24)):
        assert np.abs(rad.Fld(obj, "b", P, precision=precision) - rad.Fld(plain, "b", P, precision=precision)).max() <= tol
    M = []
    for body in (plain, obj):
        h = rad.ObjCnt([body, rad.ObjBckg([0.1, 0.2, 0.3])])
        rad.MatApl(body, mat)
        im = rad.RlxPre(h, fast=True)
        rad.RlxAuto(im, 1e-12, 200, 4)
        M.append(np.array(rad.ObjM(body)).ravel()[-3:])
    assert np.abs(M[0] - M[1]).max() <= 1e-7 and np.abs(M[0]).max() > 0.1   # the matrix is held in FP32


@pytest.mark.gpu
@pytest.mark.parametrize("current", [False, True])
@pytest.mark.parametrize("sign", [(-1, 1, 1), (1, -1, 1), (1, 1, -1), (-1, -1, 1), (-1, 1, -1), (-1, -1, -1)])
def test_negative_widths(cuda, rad, guards, sign, current):
    """The C-ABI takes cuboids of negative width: each turns the field's sign,
    as in the reference's formulas, outside and inside.  A current block
    against the positive one to the bit; against the oracle to the rounding of
    its corner terms (some 10 ulp of terms up to 4 pi |M|, and of 1e-4 times
    lengths of some 10)."""
    make = rad.ObjRecCur if current else rad.ObjRecMag
    a = _arrays(rad, make([0.1, -0.2, 0.3], [4.0, 6.0, 8.0], [0.3, -0.7, 1.1]))
    b = {k: v.copy() for k, v in a.items()}
    b["rec"][0, 3:6] *= sign
    rng = np.random.default_rng(8)
    P = np.concatenate([rng.uniform(-9, 9, size=(60, 3)), rng.uniform(-1.5, 1.5, size=(10, 3))])
    s = np.prod(sign)
    for what in (0, 1):
        got, exp = _native.field(b, P, what), O.field(b, P, what)
        if current:
            assert np.array_equal(got, s * _native.field(a, P, what))
        bound = 1e-14 if current else 1e-13
        assert np.abs(got - exp).max() <= bound
        assert np.abs(_noalloc(cuda, b, P, what) - exp).max() <= bound


CUBE = np.array([[x, y, z] for z in (0, 1) for y in (0, 1) for x in (0, 1)], float)
BODIES = {
    # axis-aligned faces meet these points exactly, so that all forms see them there
    "box": (CUBE, [[1, 3, 4, 2], [5, 6, 8, 7], [1, 2, 6, 5], [2, 4, 8, 6], [4, 3, 7, 8], [3, 1, 5, 7]]),
    "box of triangles": (CUBE, [[1, 3, 4], [1, 4, 2], [5, 6, 8], [5, 8, 7], [1, 2, 6], [1, 6, 5], [2, 4, 8], [2, 8, 6],
                                [4, 3, 7], [4, 7, 8], [3, 1, 5], [3, 5, 7]]),
    "corner": (np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]]), [[1, 2, 3], [1, 4, 2], [2, 4, 3], [3, 4, 1]]),
}


def _axis_points(name):
    """Points of the body's faces in the coordinate planes: boundary (corners
    and edges), interior, and the outward normal of each interior one."""
    t = [0.25, 0.5, 0.375]
    edge = [[0, 0, 0]] + [[a, 0, 0] for a in t] + [[0, a, 0] for a in t] + [[0, 0, a] for a in t]
    face = [[0.25, 0.375, 0], [0.375, 0, 0.25], [0, 0.25, 0.375], [0.5, 0.125, 0]]
    out = [[0, 0, -1], [0, -1, 0], [-1, 0, 0], [0, 0, -1]]
    if name != "corner":
        edge += [[1, 0, 0], [0, 1, 0], [0, 0, 1], [1, 1, 1], [1, 0, 1], [1, 1, 0.25], [0.375, 1, 1]]
        face += [[1, 0.25, 0.625], [0.25, 0.625, 1], [0.25, 1, 0.625]]
        out += [[1, 0, 0], [0, 0, 1], [0, 1, 0]]
    return np.array(edge, float), np.array(face, float), np.array(out, float)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(BODIES))
def test_points_on_polyhedra(cuda, rad, guards, name):
    """With guards the reference's values, also on edges and corners, where they
    are what its steps leave of infinite ones; next to an edge its terms lose
    half of the digits: 1e-6.  Without guards a point of a face is on its outer
    side, in B, H and M (the reference's angles cancel there: off by up to |M|,
    and even outside the body in a face's plane), and edges and corners are
    finite, as in the reference.  As one polyhedron and among others (17 units:
    more than one tile), and by the no-alloc entry."""
    V, F = BODIES[name]
    one = rad.ObjPolyhdr(V, F, [0.3, -0.7, 1.1])
    more = rad.ObjCnt([rad.ObjPolyhdr(V + [3.0 * k, 5.0, 7.0], F, [0.1, 0.2, 0.3]) for k in range(16)] +
                      [rad.ObjPolyhdr(V, F, [0.3, -0.7, 1.1])])
    edge, face, out = _axis_points(name)
    for obj in (one, more):
        arrs = _arrays(rad, obj)
        for what in (0, 1, 2):
            for run in (lambda P: _native.field(arrs, P, what), lambda P: _noalloc(cuda, arrs, P, what),
                        lambda P: _native.field(arrs, np.tile(P, (30, 1)), what)[-len(P):]):
                if guards == "on":
                    for P in (edge, face):
                        exp = O.field(arrs, P, what)
                        assert np.all(np.abs(run(P) - exp) <= 1e-6 * np.abs(exp).max(axis=1, keepdims=True) + 1e-9)
                else:
                    assert np.all(np.isfinite(run(edge)))
                    # 1e-9 off the plane the field has changed by 1e-9 of |M| / distance to an edge
                    near = run(face + 1e-9 * out)
                    assert np.abs(run(face) - near).max() <= 1e-7
                    assert what != 2 or np.all(run(face) == 0.0)
                    plane = np.array([[1.75, 0.3125, 0], [-0.5, 0.625, 0], [0, 1.375, 0.8125]])
                    assert np.abs(run(plane) - run(plane + 1e-9)).max() <= 1e-7
    # squares of these distances overflow
    for scale in (1e155, 1e160, 1e200):
        far = scale * np.array([[1.0, -0.4, 0.3]])
        assert np.array_equal(_native.field(_arrays(rad, one), far, 1), np.zeros((1, 3)))


@pytest.mark.gpu
@pytest.mark.parametrize("off", [0.0, 3e-6, -3e-6, 2e-5])
def test_points_on_an_arcs_corner_edges(cuda, rad, guards, off):
    """At a node of the arc's trapezoid rule the distances to its lower corner
    edges are not below 1e-5 in the reference; its logarithms are of the
    distances so raised.  (The upper ones it leaves as they come out of a
    cancellation, so no value there is compared.)  The oracle forms the squared
    distances by the law of cosines, 1e-15 of 1e-10: 1e-5 of a distance, in a
    logarithm of some 12 half of them; elsewhere some ulp."""
    arrs = _arrays(rad, rad.ObjArcCur([0, 0, 0], [2.0, 5.0], [0.0, 1.5], 3.0, 6, 1.7, "man", "z"))
    phi = np.arange(7) * 0.25
    P = np.array([[(r + off) * np.cos(f), (r + off) * np.sin(f), -1.5 + s * off] for r in (2.0, 5.0) for f in phi for s in (0, 1)])
    exp = O.field(arrs, P, 0)
    has = np.all(np.isfinite(exp), axis=1)   # just outside 1e-5 its sums u + D may cancel to zero
    assert has.sum() >= 14
    for got in (_native.field(arrs, P, 0), _noalloc(cuda, arrs, P, 0)):
        assert np.all(np.isfinite(got))
        assert np.abs(got - exp)[has].max() <= 1e-5 * np.abs(exp[has]).max()
    if not has[2]:
        return
    init = np.array([P[2, 0], 1e-3, P[2, 2], -1e-3])   # a trajectory that starts there
    row = np.array(rad.FldPtcTrj(rad.ObjArcCur([0, 0, 0], [2.0, 5.0], [0.0, 1.5], 3.0, 6, 1.7, "man", "z"), 0.05, init,
                                 [P[2, 1], P[2, 1] + 1.0], 3))
    ref = trajectory(lambda q: O.field(arrs, q[None], 0)[0], 0.05, init, P[2, 1], P[2, 1] + 1.0, 3)
    assert np.abs(row - ref).max() <= 1e-5 * np.abs(exp[has]).max()
