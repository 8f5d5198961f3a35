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
