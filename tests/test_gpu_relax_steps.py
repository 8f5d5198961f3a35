"""The device-resident Anderson iteration, the fused Arnoldi steps and the
triangular sweeps at sizes around their tiles (128 rows of a block or a basis
slice, 256 threads), against dense solves of the same matrix."""
import numpy as np
import pytest

import models as MD
import oracle.oracle as O
from radiacuda_b200 import _native, model
from util import rel_err


def _blocks(rad, n, sat=False):
    """n cuboids on a line, anisotropic linear or saturating in a background."""
    MD.reset(rad)
    rng = np.random.default_rng(n)
    hs = []
    iron = rad.MatSatIsoFrm([2000, 1.5], [100, 0.4], [10, 0.2])
    for k in range(n):
        m = rng.normal(size=3)
        h = rad.ObjRecMag([3.0 * k, 0.7 * (k % 3), 0.3 * (k % 5)], [2.0, 2.0, 2.0], (0 * m if sat else m).tolist())
        rad.MatApl(h, iron if sat else rad.MatLin([0.06, 0.17], m.tolist()))
        hs.append(h)
    return rad.ObjCnt(hs + [rad.ObjBckg([0.02, -0.01, 0.05])])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 42, 43, 85, 86, 171])
def test_jacobi_and_newton_reach_the_dense_solution(cuda, rad, n):
    h = _blocks(rad, n)
    pack = model.pack_interaction(rad._objs, h, 0, tuple(rad._rand))
    exp = O.linear_direct(pack, O.assemble(pack), O.extfield(pack))
    nat = _native.NativeInteraction(pack, 1)
    try:
        for method in (0, 1):
            M, H, st = nat.relax(method, 1e-13, 500, True, 1.0, np.zeros(3 * n))
            assert st[0] <= 1e-13 and 1 <= st[3] <= 500
            assert rel_err(M, exp) < 1e-11
            again, _, st2 = nat.relax(method, 1e-13, 500, True, 1.0, np.zeros(3 * n))
            assert np.array_equal(M, again) and st2[3] == st[3]   # bitwise reproducible
        # the step count is exact, in and across batches (one or two linear
        # elements reach a misfit of zero before the limit)
        for k in (1, 5, 6, 7) if n > 2 else (1,):
            _, _, st = nat.relax(0, 1e-300, k, True, 1.0, np.zeros(3 * n))
            assert st[3] == k
    finally:
        nat.free()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [7, 60])
def test_saturating_methods_agree(cuda, rad, n):
    h = _blocks(rad, n, sat=True)
    pack = model.pack_interaction(rad._objs, h, 0, tuple(rad._rand))
    nat = _native.NativeInteraction(pack, 1)
    try:
        a, _, sa = nat.relax(0, 1e-12, 3000, True, 1.0, np.zeros(3 * n))
        b, _, sb = nat.relax(1, 1e-12, 3000, True, 1.0, np.zeros(3 * n))
        # restarting from the solution ends at once
        c, _, sc = nat.relax(0, 1e-11, 3000, False, 1.0, b)
    finally:
        nat.free()
    assert sa[0] <= 1e-12 and sb[0] <= 1e-12
    assert rel_err(a, b) < 1e-9
    assert sc[3] <= 2 and rel_err(c, b) < 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("restart", [1, 2, 3, 7, 20])
@pytest.mark.parametrize("n", [86, 171])
def test_gmres_restarts(cuda, rad, n, restart, monkeypatch):
    """Newton's inner solves to 1e-10 of a strongly coupled linear system in
    cycles of a few vectors (RADB200_NK): about 35 vectors each in one cycle of
    200.  The same solution, with more products than one cycle takes, which
    only restarts add."""
    MD.reset(rad)
    rng = np.random.default_rng(n)
    hs = []
    for k in range(n):
        m = rng.normal(size=3).tolist()
        hs.append(rad.ObjRecMag([2.1 * (k % 5), 2.1 * ((k // 5) % 5), 2.1 * (k // 25)], [2.0, 2.0, 2.0], m))
        rad.MatApl(hs[-1], rad.MatLin([30.0, 18.0], m))
    h = rad.ObjCnt(hs + [rad.ObjBckg([0.02, -0.01, 0.05])])
    pack = model.pack_interaction(rad._objs, h, 0, tuple(rad._rand))
    exp = O.linear_direct(pack, O.assemble(pack), O.extfield(pack))
    nat = _native.NativeInteraction(pack, 1)
    products = {}
    try:
        for r in (200, restart):
            monkeypatch.setenv("RADB200_NK", f"1e-10,0.01,{r},5000")
            M, _, st = nat.relax(1, 1e-12, 20000, True, 1.0, np.zeros(3 * n))
            products[r] = st[3]
            assert st[0] <= 1e-12 and rel_err(M, exp) < 1e-11
    finally:
        nat.free()
    assert products[restart] > products[200] > 40


@pytest.mark.gpu
def test_newton_on_a_strongly_coupled_mesh(cuda, rad):
    """Tetrahedra of chi = 1000: several Newton steps of many vectors each."""
    h, body = MD.tet_mesh(rad, ncell=3, n_tets=100, chi=1000.0)
    pack = model.pack_interaction(rad._objs, h, 0, tuple(rad._rand))
    n = pack.elem_src.shape[0]
    exp = O.linear_direct(pack, O.assemble(pack), O.extfield(pack))
    nat = _native.NativeInteraction(pack, 1)
    try:
        M, _, st = nat.relax(1, 1e-11, 20000, True, 1.0, np.zeros(3 * n))
    finally:
        nat.free()
    assert st[0] <= 1e-11
    assert rel_err(M, exp) < 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [1, 42, 43, 85, 86, 128, 171])
def test_triangular_sweeps(cuda, rad, n, mode):
    """FP64 factors solve to their rounding in one application, FP32 ones in a
    few refinements, forward and transposed; a restored interaction forms the
    sweeps' buffers again and gives the same bits."""
    h = _blocks(rad, n)
    pack = model.pack_interaction(rad._objs, h, 0, tuple(rad._rand))
    exp = O.linear_direct(pack, O.assemble(pack), O.extfield(pack))
    g = np.random.default_rng(n + 1).normal(size=3 * n)
    nat = _native.NativeInteraction(pack, 1)
    try:
        nat.relax(1, 1e-13, 500, True, 1.0, np.zeros(3 * n))
        lam0, st0 = nat.adjoint_solve(g, 1e-13, 200)   # factors of I - D N
        M, st = nat.direct(mode, 1e-13, 60)
        lam, sa = nat.adjoint_solve(g, 1e-13, 60)      # the direct solve's own
        state = nat.save()
    finally:
        nat.free()
    # FP64 factors of these well conditioned matrices leave a residual near
    # 1e-16, so at most one refinement; FP32 ones gain at least 1e4 per step
    most = 1 if mode == 0 else 4
    assert st[0] <= 1e-13 and st[1] <= most
    assert rel_err(M, exp) < 1e-11
    assert sa[0] <= 1e-13 and sa[1] <= most + 1 and sa[2] == 1.0
    assert st0[0] <= 1e-13 and rel_err(lam, lam0) < 1e-11
    again = _native.NativeInteraction(pack, 1, state)
    try:
        lam2, _ = again.adjoint_solve(g, 1e-13, 60)
    finally:
        again.free()
    assert np.array_equal(lam2, lam)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [86, 171, 300])
def test_a_sweep_whose_wait_runs_out_ends(cuda, rad, n, mode, monkeypatch):
    """RADB200_SWEEP_SPIN=0: blocks after the first give up at once, with the
    copies of their inverses under way.  The solve fails, the device goes on."""
    h = _blocks(rad, n)
    pack = model.pack_interaction(rad._objs, h, 0, tuple(rad._rand))
    nat = _native.NativeInteraction(pack, 1)
    try:
        monkeypatch.setenv("RADB200_SWEEP_SPIN", "0")
        with pytest.raises(Exception):
            nat.direct(mode, 1e-13, 60)
    finally:
        monkeypatch.undo()
        nat.free()
    P = np.array([[0.317, 5.071, 0.233]])
    g = model.pack_sources(rad._objs, h, tuple(rad._rand))
    assert rel_err(_native.field(g, P, 0), O.field(g, P, 0)) < 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1])
def test_a_sweep_time_out_is_reported_and_forgotten(cuda, rad, mode, monkeypatch):
    """The direct and the adjoint solve name the time-out, and the next solves,
    on this interaction and on another, give what they gave before it."""
    h = _blocks(rad, 171)
    pack = model.pack_interaction(rad._objs, h, 0, tuple(rad._rand))
    g = np.random.default_rng(3).normal(size=3 * 171)
    nat, other = _native.NativeInteraction(pack, 1), _native.NativeInteraction(pack, 1)
    try:
        M = nat.direct(mode, 1e-13, 60)[0].copy()
        lam = nat.adjoint_solve(g, 1e-13, 60)[0].copy()
        for k in range(2):
            monkeypatch.setenv("RADB200_SWEEP_SPIN", "0")
            with pytest.raises(Exception, match="timed out"):
                nat.adjoint_solve(g, 1e-13, 60)
            if k:
                with pytest.raises(Exception, match="timed out"):
                    nat.direct(mode, 1e-13, 60)
            monkeypatch.delenv("RADB200_SWEEP_SPIN")
            assert np.array_equal(other.direct(mode, 1e-13, 60)[0], M)
            assert np.array_equal(nat.direct(mode, 1e-13, 60)[0], M)
            assert np.array_equal(nat.adjoint_solve(g, 1e-13, 60)[0], lam)
    finally:
        nat.free()
        other.free()
