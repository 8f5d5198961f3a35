"""Performance cases of the relaxation path, through the public Python API.

Each case is one thing that a Radia program has the library do: a field
evaluation (rad.Fld), a relaxation (rad.Solve, or rad.RlxPre + rad.RlxAuto), an
electron trajectory (rad.FldPtcTrj) or a gradient through the relaxation
(adjoint.FieldProblem).  Models are the shapes of this repository's benchmark
and tests: a permanent-magnet array, an iron dipole with mirror planes and a
racetrack coil, tetrahedral meshes, a planar and a hybrid undulator.

listed() gives the fixed cases, draw(rng) more of the same ranges; prepare()
builds a model (what a program holds before the call), run() makes the call,
exact() evaluates the same quantity in 64 bits with plain torch and numpy.
"""
import math

import numpy as np
import torch

from radiacuda_b200 import adjoint, rad

TET_FACES = [[1, 2, 3], [1, 4, 2], [2, 4, 3], [3, 4, 1]]
CUBE = [[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]]
KUHN = [[0, 1, 2, 6], [0, 2, 3, 6], [0, 3, 7, 6], [0, 7, 4, 6], [0, 4, 5, 6], [0, 5, 1, 6]]
TET_EDGE = 2.0


def listed():
    return [
        # a script that looks at one point of a magnet assembly: the smallest call
        dict(name="field_one_point", kind="field_magnets", nside=4, div=3, npts=1),
        # the field map of the 432-block magnet array over its 10,000-point grid
        dict(name="field_magnets", kind="field_magnets", nside=4, div=3, npts=10000),
        # the gap field of an iron dipole: four symmetry images and a racetrack coil
        dict(name="field_dipole", kind="field_dipole", nelem=4000, npts=250000),
        # a field map of a tetrahedral mesh with FP32 terms (precision='single')
        dict(name="field_tets_single", kind="field_tets", ntets=8000, npts=1000000, precision="single"),
        # the same in the default precision (the polygon faces one by one)
        dict(name="field_tets_double", kind="field_tets", ntets=3000, npts=20000, precision="double"),
        # and in FP64 by vertices and edges (precision='fast')
        dict(name="field_tets_fast", kind="field_tets", ntets=6000, npts=100000, precision="fast"),
        # relaxation of the small magnet array, as a design loop repeats it
        dict(name="solve_magnets", kind="solve_magnets", nside=4, div=3, meth=4),
        # relaxation of the saturating dipole yoke with its coil
        dict(name="solve_dipole", kind="solve_dipole", nelem=4000, meth=4),
        # dense direct solve of a tetrahedral iron body, mixed precision: the headline system
        dict(name="solve_tets", kind="solve_tets", ntets=20000),
        # one forward and one backward pass of a shimming optimization (linear materials)
        dict(name="grad_undulator", kind="grad_undulator", nper_row=40, div=2, npts=4000),
        # the same through a saturating hybrid undulator (Newton-Krylov forward solve)
        dict(name="grad_hybrid", kind="grad_hybrid", npairs=40, pole=4, npts=50000),
        # an electron tracked through the dipole's gap
        dict(name="trajectory", kind="trajectory", nelem=300, npts=401, ntraj=1),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["field_magnets", "field_magnets", "field_dipole", "field_tets", "field_tets", "field_tets",
                       "solve_magnets", "solve_dipole", "solve_tets", "grad_undulator", "grad_hybrid", "trajectory"])
    c = dict(kind=kind)
    if kind == "field_magnets":
        c.update(nside=rng.randint(1, 8), div=rng.randint(1, 4), npts=_logint(rng, 1, 40000))
    elif kind == "field_dipole":
        n = _logint(rng, 20, 4000)
        c.update(nelem=n, npts=_logint(rng, 10, 250000))
    elif kind == "field_tets":
        prec = rng.choice(["single", "double", "fast"])
        n = _logint(rng, 5, 6000)
        most = {"single": 8e8, "double": 6e7, "fast": 6e8}[prec]
        c.update(ntets=n, npts=_logint(rng, 1, max(2, min(500000, int(most / n)))), precision=prec)
    elif kind == "solve_magnets":
        c.update(nside=rng.randint(1, 8), div=rng.randint(1, 4), meth=rng.choice([4, 11]))
    elif kind == "solve_dipole":
        c.update(nelem=_logint(rng, 50, 4000), meth=rng.choice([4, 4, 11]))
    elif kind == "solve_tets":
        c.update(ntets=_logint(rng, 40, 9000))
    elif kind == "grad_undulator":
        c.update(nper_row=rng.randint(3, 60), div=rng.randint(1, 2), npts=_logint(rng, 50, 5000))
    elif kind == "grad_hybrid":
        c.update(npairs=rng.randint(2, 24), pole=rng.randint(2, 4), npts=_logint(rng, 100, 30000))
    else:
        c.update(nelem=_logint(rng, 50, 600), npts=_logint(rng, 11, 301), ntraj=rng.choice([1, 1, 3, 40]))
    return c


# ---------------------------------------------------------------------------
# models: plain arrays (used by exact() too) and the rad objects built from them
# ---------------------------------------------------------------------------
def _unit(rng, n):
    v = rng.normal(size=(n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _split(c, d, k):
    """Centres and dimensions of the k[0] x k[1] x k[2] equal parts, x slowest."""
    c, d = np.asarray(c, float), np.asarray(d, float)
    s = d / np.asarray(k)
    g = np.meshgrid(*[np.arange(q) for q in k], indexing="ij")
    i = np.stack([x.ravel() for x in g], axis=1)
    return c - 0.5 * d + (i + 0.5) * s, np.repeat(s[None], len(i), axis=0)


def _magnets(case, seed):
    """nside x nside NdFeB blocks of 10 mm, div^3 parts each."""
    rng = np.random.default_rng(seed)
    n, div = case["nside"], case["div"]
    c = np.array([[-6.0 * (n - 1) + 12.0 * i, -6.0 * (n - 1) + 12.0 * j, 0.0] for i in range(n) for j in range(n)])
    mr = rng.uniform(1.1, 1.3) * _unit(rng, n * n)
    half = 6.0 * n - 1.0
    m = max(1, case.get("npts", 1))
    k = max(1, int(math.ceil((m / 16.0) ** 0.5)))
    x = np.linspace(-half, half, k) + rng.uniform(0.1, 0.2)
    z = np.linspace(10, 25, 16) + rng.uniform(0.03, 0.07)
    P = np.stack([a.ravel() for a in np.meshgrid(x, x, z, indexing="ij")], axis=1)[:m]
    blocks = [dict(c=c[b], d=[10.0] * 3, k=[div] * 3, mr=mr[b], mat=("lin", 0.06, 0.17)) for b in range(n * n)]
    return blocks, np.ascontiguousarray(P)


def _dipole(case, seed):
    """C-shaped yoke of saturating iron in the quadrant x, z > 0, about nelem
    cuboids, mirrored at x = 0 and z = 0, with a racetrack coil."""
    rng = np.random.default_rng(seed)
    hg = 20.0
    # widths without common divisors and a coil a little off centre: element
    # centres stay off the other sources' face planes, where the closed forms are singular
    parts = [([15.0, 0.0, hg + 20.0], [30.0, 80.0, 40.0]), ([50.65, 0.37, hg + 55.0], [101.3, 80.0, 30.0]),
             ([85.0, -0.53, 29.95], [29.9, 80.0, 59.9])]
    h = (sum(np.prod(d) for _, d in parts) / case["nelem"]) ** (1.0 / 3.0)
    mat = ("sat", [20000.0, 2.0], [0.1, 2.0], [0.1, 2.0])
    blocks = [dict(c=c, d=d, k=[max(1, int(round(x / h))) for x in d], mr=[0.0] * 3, mat=mat) for c, d in parts]
    coil = dict(P=list(np.array([0.0, 0.0, hg + 20.0]) + rng.uniform(0.03, 0.3, 3)), R=[2.0, 22.0], L=[60.0, 80.0], h=30.0, nseg=6,
                j=rng.uniform(0.9, 1.1) * 10000.0 / 600.0)
    return blocks, coil, rng


def _grid_in_gap(n, rng):
    k = max(1, int(math.ceil(n ** (1.0 / 3.0))))
    x = np.linspace(-45, 45, k) + rng.uniform(0.1, 0.2)
    z = np.linspace(-18, 18, k) + rng.uniform(0.03, 0.07)
    return np.ascontiguousarray(np.stack([a.ravel() for a in np.meshgrid(x, x, z, indexing="ij")], axis=1)[:n])


DIPOLE_IMAGES = [((1, 1, 1), 1.0), ((1, 1, -1), -1.0), ((-1, 1, 1), 1.0), ((-1, 1, -1), -1.0)]


def _tet_vertices(n, rng):
    """n tetrahedra [n, 4, 3] of a jittered lattice of cubes, 2% of them slivers."""
    ncell = max(1, int(math.ceil((n / 6.0) ** (1.0 / 3.0))))
    g = ncell + 1
    P = np.stack([a.ravel() for a in np.meshgrid(*[np.arange(g)] * 3, indexing="ij")], axis=1) * TET_EDGE
    P = P + rng.uniform(-0.02, 0.02, size=P.shape) * TET_EDGE
    cell = np.stack([a.ravel() for a in np.meshgrid(*[np.arange(ncell)] * 3, indexing="ij")], axis=1)
    corner = cell[:, None, :] + np.array(CUBE)[None]                       # [cells, 8, 3]
    idx = (corner[..., 0] * g + corner[..., 1]) * g + corner[..., 2]
    V = P[idx[:, np.array(KUHN)].reshape(-1, 4)[:n]].copy()
    for s in rng.choice(n, size=int(round(0.02 * n)), replace=False):
        c = V[s, :3].mean(axis=0)
        V[s, 3] = c + (V[s, 3] - c) * rng.uniform(0.02, 0.2)
    return V, ncell * TET_EDGE


def _points_outside(n, L, rng, margin=2.0):
    lo, hi = -margin - 0.25 * L - 1.0, L + margin + 0.25 * L + 1.0
    out = np.empty((0, 3))
    while out.shape[0] < n:
        p = rng.uniform(lo, hi, size=(2 * n + 16, 3))
        out = np.concatenate([out, p[~np.all((p > -margin) & (p < L + margin), axis=1)]])
    return np.ascontiguousarray(out[:n])


def _tets(case, seed):
    rng = np.random.default_rng(seed)
    V, L = _tet_vertices(case["ntets"], rng)
    M = 1.3 * _unit(rng, 1) + 0.2 * rng.normal(size=(len(V), 3))
    return V, M, _points_outside(case.get("npts", 1), L, rng)


def _undulator(case, seed):
    """Two rows of 50 x 10 x 5 mm blocks, M turning by 90 degrees per block."""
    rng = np.random.default_rng(seed)
    n, div = case["nper_row"], case["div"]
    blocks = []
    for row in (1, -1):
        for k in range(n):
            d = np.array([(0, 1, 0), (0, 0, row), (0, -1, 0), (0, 0, -row)][k % 4], float) * row
            mr = 1.3 * (1.0 + 0.02 * rng.uniform(-1, 1)) * (d + 0.01 * rng.normal(size=3))
            blocks.append(dict(c=np.array([0.0, row * 10.0, (k - 0.5 * (n - 1)) * 5.0]), d=[50.0, 10.0, 5.0],
                               k=[div] * 3, mr=mr, mat=("lin", 0.05, 0.15)))
    z = np.linspace(-2.5 * n, 2.5 * n, case["npts"]) + 0.0517
    P = np.stack([np.full(len(z), 0.1371), np.full(len(z), 0.0913), z], axis=1)
    return blocks, P, rng.normal(size=P.shape)


def _hybrid(case, seed):
    """NdFeB blocks between saturating poles, mirrored at y = 0."""
    rng = np.random.default_rng(seed)
    n, kp = case["npairs"], case["pole"]
    poles, magnets = [], []
    for k in range(n):
        zp = -5.0 * n + 10.0 * k + 2.0
        poles.append(dict(c=[0.0, 15.0, zp], d=[40.0, 20.0, 4.0], k=[kp] * 3, mr=[0.0] * 3,
                          mat=("sat", [2000.0, 1.5], [100.0, 0.4], [10.0, 0.2])))
        mr = np.array([0.0, 0.0, 1.25 if k % 2 == 0 else -1.25]) * (1.0 + 0.01 * rng.uniform(-1, 1))
        magnets.append(dict(c=[0.0, 18.0, zp + 5.0], d=[50.0, 25.0, 6.0], k=[2, 2, 3], mr=mr, mat=("lin", 0.05, 0.15)))
    L = 5.0 * n
    P = rng.uniform([-15, -4, -L], [15, 4, L], size=(case["npts"], 3)) + np.array([0.0137, 0.0071, 0.0517])
    return poles + magnets, P, rng.normal(size=P.shape)


HYBRID_IMAGES = [((1, 1, 1), 1.0), ((1, -1, 1), -1.0)]


class _Model:
    """The rad objects of one prepared state; they go with it."""

    def __init__(self):
        self.handles = []

    def add(self, h):
        self.handles.append(h)
        return h

    def __del__(self):
        if rad is None:  # the interpreter is going down
            return
        for h in self.handles:
            for m in rad._objs[h].members if h in rad._objs and hasattr(rad._objs[h], "members") else ():
                rad.UtiDel(m)
            rad.UtiDel(h)


def _material(m, mr):
    if m[0] == "lin":
        return rad.MatLin([m[1], m[2]], list(mr))
    return rad.MatSatIsoFrm(*[list(p) for p in m[1:]])


def _build_blocks(M, blocks):
    """A container of the blocks, each subdivided and with its material."""
    hs = []
    sat = {}
    for b in blocks:
        h = M.add(rad.ObjRecMag(list(b["c"]), list(b["d"]), list(b["mr"])))
        if b["mat"][0] == "lin":
            rad.MatApl(h, M.add(_material(b["mat"], b["mr"])))
        else:
            key = repr(b["mat"])
            if key not in sat:
                sat[key] = M.add(_material(b["mat"], b["mr"]))
            rad.MatApl(h, sat[key])
        if b["k"] != [1, 1, 1]:
            rad.ObjDivMag(h, b["k"])
        hs.append(h)
    return M.add(rad.ObjCnt(hs))


def _build_dipole(M, blocks, coil):
    yoke = _build_blocks(M, blocks)
    rad.TrfZerPerp(yoke, [0, 0, 0], [1, 0, 0])
    rad.TrfZerPara(yoke, [0, 0, 0], [0, 0, 1])
    c = M.add(rad.ObjRaceTrk(coil["P"], coil["R"], coil["L"], coil["h"], coil["nseg"], coil["j"], "man", "z"))
    return M.add(rad.ObjCnt([yoke, c])), yoke


def _yoke_m(blocks, seed):
    """A plausible magnetization of the yoke for the field cases."""
    E = _elements(blocks)
    rng = np.random.default_rng(seed + 1)
    c = E["c"]
    return 1.5 * np.stack([c[:, 2] - 40.0, 0.1 * c[:, 1], 60.0 - c[:, 0]], axis=1) / 60.0 + 0.05 * rng.normal(size=c.shape)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    rad.FldLenRndSw("off")
    kind = case["kind"]
    M = _Model()
    s = dict(case=case, model=M)
    if kind in ("field_magnets", "solve_magnets"):
        blocks, P = _magnets(case, seed)
        s.update(obj=_build_blocks(M, blocks), pts=P)
        if case.get("npts") == 1:
            s["pts"] = P[0].tolist()
    elif kind in ("field_dipole", "solve_dipole", "trajectory"):
        blocks, coil, rng = _dipole(case, seed)
        s["obj"], yoke = _build_dipole(M, blocks, coil)
        if kind != "solve_dipole":
            for h, m in zip([q for b in rad.ObjCntStuf(yoke) for q in rad.ObjCntStuf(b)], _yoke_m(blocks, seed)):
                rad.ObjSetM(h, m)
        if kind == "field_dipole":
            s["pts"] = _grid_in_gap(case["npts"], rng)
        elif kind == "trajectory":
            s["init"] = _beam(case, rng)
    elif kind == "field_tets":
        V, Mg, P = _tets(case, seed)
        s.update(obj=M.add(rad.ObjCnt([rad.ObjPolyhdr(v, TET_FACES, m) for v, m in zip(V, Mg)])), pts=P)
    elif kind == "solve_tets":
        V, _, _ = _tets(case, seed)
        body = M.add(rad.ObjCnt([rad.ObjPolyhdr(v, TET_FACES) for v in V]))
        rad.MatApl(body, M.add(rad.MatLin([1000.0, 1000.0], [0, 0, 1e-12])))
        s["obj"] = M.add(rad.ObjCnt([body, M.add(rad.ObjBckg(_background(seed)))]))
    else:
        blocks, P, W = (_undulator if kind == "grad_undulator" else _hybrid)(case, seed)
        obj = _build_blocks(M, blocks)
        if kind == "grad_hybrid":
            rad.TrfZerPara(obj, [0, 0, 0], [0, 1, 0])
        s.update(problem=adjoint.FieldProblem(obj, P), W=W)
    return s


def _background(seed):
    return (np.array([0.0, 0.0, 1.0]) + 0.2 * np.random.default_rng(seed + 7).normal(size=3)).tolist()


def _beam(case, rng):
    """Electrons entering the gap along y: x, x', z, z' (mm, rad)."""
    n = case.get("ntraj", 1)
    a = rng.uniform([-3, -0.002, -3, -0.002], [3, 0.002, 3, 0.002], size=(n, 4))
    return a[0] if n == 1 else a


BEAM = (0.3, [-120.0, 119.7])  # GeV; y range (mm)


def _positions_and_angles(r):
    """The rows (y, x, x', z, z') by unit, so that each is compared on its own scale."""
    return dict(y=r[..., 0], position=r[..., (1, 3)], angle=r[..., (2, 4)])


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("field_magnets", "field_dipole"):
        return np.asarray(rad.Fld(s["obj"], "b", s["pts"]))
    if kind == "field_tets":
        return rad.Fld(s["obj"], "b", s["pts"], precision=case["precision"])
    if kind == "trajectory":
        return _positions_and_angles(np.asarray(rad.FldPtcTrj(s["obj"], BEAM[0], s["init"], BEAM[1], case["npts"])))
    if kind in ("grad_undulator", "grad_hybrid"):
        p = s["problem"]
        F = p.forward()
        g = p.backward(s["W"])
        return dict(F=F, M=p.magnetization, **g)
    if kind == "solve_tets":
        im = rad.RlxPre(s["obj"], storage="mixed", fast=True)
        rad.RlxAuto(im, 1e-13, 200, 13)
    else:
        im = rad.RlxPre(s["obj"])
        rad.RlxAuto(im, 1e-10 if kind == "solve_magnets" else 1e-7, 5000, case["meth"])
    M = rad._objs[im].M.reshape(-1, 3)
    rad.UtiDel(im)
    return M


# ---------------------------------------------------------------------------
# the work that a pass cannot do without
# ---------------------------------------------------------------------------
# operations of one pair in the closed forms (adds, multiplications, and 20 for
# each root, logarithm, arctangent or division): a cuboid's 8 corners give 8
# roots, 3 logarithms of ratios and 3 arctangents of products, plus the
# products themselves; a tetrahedron 4 roots, 6 logarithms, 4 solid angles
PAIR = {"cuboid": 560.0, "tet": 541.0}


def work(case):
    kind = case["kind"]
    if kind in ("field_magnets", "solve_magnets"):
        n, images = (case["nside"] * case["div"]) ** 2 * case["div"], 1
    elif kind in ("field_dipole", "solve_dipole", "trajectory"):
        n, images = len(_elements(_dipole(case, 0)[0])["c"]), 4
    elif kind in ("field_tets", "solve_tets"):
        n, images = case["ntets"], 1
    elif kind == "grad_undulator":
        n, images = 2 * case["nper_row"] * case["div"] ** 3, 1
    else:
        n, images = case["npairs"] * (case["pole"] ** 3 + 12), 2
    per = PAIR["tet" if "tets" in kind else "cuboid"]
    rec = 96.0 * n
    if kind.startswith("field"):
        return dict(bytes=rec + 48.0 * case["npts"], flops=per * n * images * case["npts"])
    if kind == "trajectory":
        stages = case["ntraj"] * 4.0 * (case["npts"] - 1)
        return dict(bytes=rec + 40.0 * case["npts"] * case["ntraj"], flops=per * n * images * stages)
    n3 = 3.0 * n
    asm = per * n * n * images
    if kind == "solve_tets":
        return dict(bytes=4 * n3 * n3 * 2, flops=asm + 2.0 / 3.0 * n3 ** 3)
    if kind.startswith("solve"):
        return dict(bytes=4 * n3 * n3, flops=asm + 2 * n3 * n3)
    dense = 2.0 / 3.0 * n3 ** 3 if kind == "grad_undulator" else 2 * n3 * n3
    return dict(bytes=8 * n3 * n3 + 72.0 * case["npts"], flops=2 * asm + dense + 3 * per * n * images * case["npts"])


def tolerance(case):
    kind = case["kind"]
    if kind == "field_tets":
        # FP32 terms against the FP64 sums; FP64: rounding of the closed forms, which the distance amplifies
        return {"rel": 4e-6, "max": 5e-4} if case["precision"] == "single" else {"rel": 7e-9, "max": 1e-6}
    if kind in ("field_magnets", "field_dipole"):
        return {"rel": 1e-10, "max": 1e-8}
    if kind == "trajectory":
        return {"rel": 1e-9, "max": 1e-7}
    if kind == "solve_magnets":
        return {"rel": 1e-7, "max": 1e-5}   # the matrix is held in FP32
    if kind == "solve_dipole":
        return {"rel": 1e-4, "max": 1e-2}   # FP32 matrix and the stopping misfit, amplified by the soft iron
    if kind == "solve_tets":
        return {"rel": 1e-8, "max": 1e-6}
    return {"rel": 1e-7, "max": 1e-5} if kind == "grad_undulator" else {"rel": 1e-6, "max": 1e-4}


# ---------------------------------------------------------------------------
# the same quantities in 64 bits
# ---------------------------------------------------------------------------
DEV = "cuda" if torch.cuda.is_available() else "cpu"
F4PI = 1.0 / (4.0 * math.pi)


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=DEV)


def _elements(blocks):
    """Sub-blocks of all blocks in order: centres, dimensions, remanences, materials."""
    c, d, mr, mats = [], [], [], []
    for b in blocks:
        cc, dd = _split(b["c"], b["d"], b["k"])
        c.append(cc)
        d.append(dd)
        mr.append(np.repeat(np.asarray(b["mr"], float)[None], len(cc), axis=0))
        mats += [b["mat"]] * len(cc)
    return dict(c=np.concatenate(c), d=np.concatenate(d), mr=np.concatenate(mr), mats=mats)


def _corners(q, h):
    """Offsets and distances of the 8 corners with their signs; q, h [..., 3]."""
    for ex in (1.0, -1.0):
        for ey in (1.0, -1.0):
            for ez in (1.0, -1.0):
                X, Y, Z = q[..., 0] - ex * h[..., 0], q[..., 1] - ey * h[..., 1], q[..., 2] - ez * h[..., 2]
                yield ex * ey * ez, X, Y, Z, torch.sqrt(X * X + Y * Y + Z * Z)


def _cuboid_tensor(q, h):
    """Six entries (xx, yy, zz, xy, xz, yz) of H per unit M of a cuboid at q from its centre."""
    T = [0.0] * 6
    for p, X, Y, Z, R in _corners(q, h):
        T[0] = T[0] + p * torch.atan(Y * Z / (X * R))
        T[1] = T[1] + p * torch.atan(X * Z / (Y * R))
        T[2] = T[2] + p * torch.atan(X * Y / (Z * R))
        T[3] = T[3] - p * torch.asinh(Z / torch.sqrt(X * X + Y * Y))
        T[4] = T[4] - p * torch.asinh(Y / torch.sqrt(X * X + Z * Z))
        T[5] = T[5] - p * torch.asinh(X / torch.sqrt(Y * Y + Z * Z))
    return [F4PI * x for x in T]


def _apply6(T, m):
    return torch.stack([T[0] * m[..., 0] + T[3] * m[..., 1] + T[4] * m[..., 2],
                        T[3] * m[..., 0] + T[1] * m[..., 1] + T[5] * m[..., 2],
                        T[4] * m[..., 0] + T[5] * m[..., 1] + T[2] * m[..., 2]], dim=-1)


def _blocks_field(P, c, d, m, images, want_b=True):
    """B (or H) at P [p, 3] of cuboids with magnetization m, over symmetry images."""
    out = torch.zeros_like(P)
    for r, s in images:
        r = _t(r)
        q = (P * r)[:, None, :] - c[None]
        H = _apply6(_cuboid_tensor(q, 0.5 * d[None].expand_as(q)), m[None])
        if want_b:
            H = H + torch.where((q.abs() < 0.5 * d[None]).all(-1, keepdim=True), m[None], torch.zeros_like(H))
        out = out + s * r * H.sum(1)
    return out


def _chunked(f, P, n):
    step = max(1, int(6e6 // max(n, 1)))
    return torch.cat([f(P[i:i + step]) for i in range(0, P.shape[0], step)])


def _current_block(P, c, d, J):
    """B of a cuboid with current density J (A/mm^2): 1e-4 J x int r/|r|^3 dV."""
    v = [0.0] * 3
    h = 0.5 * d
    for p, X, Y, Z, R in _corners(P - c, h.expand_as(P)):
        x = [X, Y, Z]
        for a in range(3):
            A, B, C = x[a], x[(a + 1) % 3], x[(a + 2) % 3]
            v[a] = v[a] + p * (B * torch.asinh(C / torch.sqrt(A * A + B * B)) + C * torch.asinh(B / torch.sqrt(A * A + C * C))
                               - A * torch.atan(B * C / (A * R)))
    v = torch.stack(v, dim=-1)
    return 1e-4 * torch.linalg.cross(J.expand_as(v), v)


def _arc(P, c, R, phi, h, j, nseg):
    """B of an arc current, trapezoid rule over nseg sectors in phi."""
    p = P - _t(c)
    tiny = 1e-10
    r = torch.sqrt(p[:, 0] ** 2 + p[:, 1] ** 2 + tiny)
    f0 = torch.acos(p[:, 0] / r)
    f0 = torch.where(p[:, 1] < 0, 2 * math.pi - f0, f0)
    z = [-0.5 * h - p[:, 2], 0.5 * h - p[:, 2]]
    step = (phi[1] - phi[0] + tiny) / nseg
    out = torch.zeros_like(P)
    for i in range(nseg + 1):
        a = phi[0] - f0 + tiny + i * step
        rc, rs = r * torch.cos(a), r * torch.sin(a).abs()
        xy = torch.zeros_like(r)
        zz = torch.zeros_like(r)
        # cross-section integral, corners (radius u = R_k - r cos, height z_l)
        for k, sk in ((0, -1.0), (1, 1.0)):
            u = R[k] - rc
            for l, sl in ((0, -1.0), (1, 1.0)):
                D = torch.sqrt(u * u + rs * rs + z[l] * z[l])
                lu = torch.asinh(u / torch.sqrt(rs * rs + z[l] * z[l]))
                lz = torch.asinh(z[l] / torch.sqrt(u * u + rs * rs))
                xy = xy + sk * sl * (D + rc * lu)
                zz = zz + sk * sl * (z[l] * lu - rc * lz - rs * torch.atan(u * z[l] / (rs * D)))
        w = 0.5 if i in (0, nseg) else 1.0
        out += w * torch.stack([torch.cos(a + f0) * xy, torch.sin(a + f0) * xy, zz], dim=-1)
    return 1e-4 * j * step * out


def _coil_field(P, k):
    """B of the racetrack: four arcs and four straight blocks."""
    c, R, L, h, j = k["P"], k["R"], k["L"], k["h"], k["j"]
    out = torch.zeros_like(P)
    pi = math.pi
    for sx, sy, a, b in ((1, 1, 0.0, 0.5 * pi), (-1, 1, 0.5 * pi, pi), (-1, -1, pi, 1.5 * pi),
                         (1, -1, 1.5 * pi, 1.999999999999 * pi)):
        out = out + _arc(P, [c[0] + 0.5 * sx * L[0], c[1] + 0.5 * sy * L[1], c[2]], R, (a, b), h, j, k["nseg"])
    w = R[1] - R[0]
    for s in (1.0, -1.0):
        e = 0.5 * (L[0] + R[0] + R[1])
        out = out + _current_block(P, _t([c[0] + s * e, c[1], c[2]]), _t([w, L[1], h]), _t([0.0, s * j, 0.0]))
        e = 0.5 * (L[1] + R[0] + R[1])
        out = out + _current_block(P, _t([c[0], c[1] + s * e, c[2]]), _t([L[0], w, h]), _t([-s * j, 0.0, 0.0]))
    return out


EDGES = ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))
FACES = ((1, 2, 3), (0, 2, 3), (0, 1, 3), (0, 1, 2))


def _tet_terms(V):
    """Outward unit normals [n, 4, 3] and, per (edge, face), the outward in-plane edge normals."""
    cen = V.mean(1)
    nrm, nu = [], {}
    for f, (a, b, c) in enumerate(FACES):
        n = torch.linalg.cross(V[:, b] - V[:, a], V[:, c] - V[:, a])
        n = n / n.norm(dim=-1, keepdim=True)
        n = torch.where(((V[:, a] - cen) * n).sum(-1, keepdim=True) < 0, -n, n)
        nrm.append(n)
        fc = (V[:, a] + V[:, b] + V[:, c]) / 3.0
        for e, (i, j) in enumerate(EDGES):
            if i in (a, b, c) and j in (a, b, c):
                u = torch.linalg.cross((V[:, j] - V[:, i]) / (V[:, j] - V[:, i]).norm(dim=-1, keepdim=True), n)
                nu[e, f] = torch.where(((V[:, i] - fc) * u).sum(-1, keepdim=True) < 0, -u, u)
    return torch.stack(nrm, 1), nu


def _tet_scalars(P, V, nrm):
    """Edge logarithms [6] and signed solid angles [4] of tetrahedra at points, each [p, n]."""
    r = V[None] - P[:, None, None, :]
    R = r.norm(dim=-1)
    L, W = [], []
    for i, j in EDGES:
        l = (V[:, i] - V[:, j]).norm(dim=-1)[None]
        s = (r[:, :, i] * r[:, :, j]).sum(-1)
        D = torch.where(s > 0, R[..., i] * R[..., j] + s,
                        torch.linalg.cross(r[:, :, i], r[:, :, j]).square().sum(-1) / (R[..., i] * R[..., j] - s))
        L.append(torch.log1p(l * (R[..., i] + R[..., j] + l) / D))
    for f, (a, b, c) in enumerate(FACES):
        m = torch.linalg.cross(V[:, b] - V[:, a], V[:, c] - V[:, a])
        m = m * torch.sign((m * nrm[:, f]).sum(-1, keepdim=True))
        num = (r[:, :, a] * m[None]).sum(-1)
        den = R[..., a] * R[..., b] * R[..., c] + (r[:, :, a] * r[:, :, b]).sum(-1) * R[..., c] \
            + (r[:, :, a] * r[:, :, c]).sum(-1) * R[..., b] + (r[:, :, b] * r[:, :, c]).sum(-1) * R[..., a]
        W.append(2.0 * torch.atan2(-num, den))
    return L, W


def _tets_field(P, V, m, terms):
    """B at points outside the tetrahedra."""
    nrm, nu = terms
    sig = (nrm * m[:, None]).sum(-1)                       # [n, 4]
    L, W = _tet_scalars(P, V, nrm)
    out = torch.zeros_like(P)
    for f in range(4):
        out = out + W[f] @ (sig[:, f, None] * nrm[:, f])
    for e in range(6):
        g = sum(sig[:, f, None] * nu[k, f] for (k, f) in nu if k == e)
        out = out + L[e] @ g
    return F4PI * out


def _tets_matrix(V, terms):
    nrm, nu = terms
    n = V.shape[0]
    P = V.mean(1)
    N = torch.empty((n, 3, n, 3), dtype=torch.float64, device=V.device)
    step = max(1, int(4e6 // n))
    for i in range(0, n, step):
        L, W = _tet_scalars(P[i:i + step], V, nrm)
        B = sum(W[f][..., None, None] * (nrm[:, f, :, None] * nrm[:, f, None, :])[None] for f in range(4))
        for (e, f), u in nu.items():
            B = B + L[e][..., None, None] * (u[:, :, None] * nrm[:, f, None, :])[None]
        N[i:i + step] = F4PI * B.permute(0, 2, 1, 3)
    return N.reshape(3 * n, 3 * n)


def _blocks_matrix(P, c, d, images):
    """H at P [p, 3] per unit M of each cuboid, all images: [3p, 3n], differentiable."""
    out = 0.0
    for r, s in images:
        r = _t(r)
        q = (P * r)[:, None, :] - c[None]
        T = _cuboid_tensor(q, 0.5 * d[None].expand_as(q))
        B = torch.stack([torch.stack([T[0], T[3], T[4]], -1), torch.stack([T[3], T[1], T[5]], -1),
                         torch.stack([T[4], T[5], T[2]], -1)], -2)           # [p, n, 3, 3]
        out = out + s * r[None, None, :, None] * B
    return out.permute(0, 2, 1, 3).reshape(3 * P.shape[0], 3 * c.shape[0])


def _law(mats, mr):
    """M(H) and dM/dH of all elements; linear tensors as (chi, Mr)."""
    n = len(mats)
    lin = np.array([m[0] == "lin" for m in mats])
    chi = np.zeros((n, 3, 3))
    K, S = np.zeros((n, 3)), np.ones((n, 3))
    for e, m in enumerate(mats):
        if m[0] == "lin":
            a = mr[e] / np.linalg.norm(mr[e])
            chi[e] = m[2] * np.eye(3) + (m[1] - m[2]) * np.outer(a, a)
        else:
            for k, (ks, ms) in enumerate(m[1:]):
                K[e, k], S[e, k] = ks, ms
    chi, K, S, Mr, lin = _t(chi), _t(K), _t(S), _t(np.where(lin[:, None], mr, 0.0)), torch.as_tensor(lin, device=DEV)

    def law(H):
        h = H.norm(dim=-1).clamp_min(1e-12)
        t = torch.tanh(K * h[:, None] / S)
        f, df = (S * t).sum(-1), (K * (1 - t * t)).sum(-1)
        u = H / h[:, None]
        uu = u[:, :, None] * u[:, None, :]
        eye = torch.eye(3, dtype=H.dtype, device=H.device)[None]
        M = torch.where(lin[:, None], (chi @ H[..., None])[..., 0] + Mr, f[:, None] * u)
        D = torch.where(lin[:, None, None], chi, df[:, None, None] * uu + (f / h)[:, None, None] * (eye - uu))
        Xs = torch.where(lin[:, None, None], chi, (f / h)[:, None, None] * eye)
        return M, D, Xs

    return law, chi, Mr


def _relax(N, Hext, law, Mr):
    """H of the relaxed state and its relative residual: secant steps, then
    Newton with a line search, both with dense solves."""
    n = Hext.shape[0]
    N4 = N.reshape(3 * n, n, 3)
    eye = torch.eye(3 * n, dtype=N.dtype, device=N.device)
    drive = Hext.reshape(-1) + N @ Mr.reshape(-1)

    def residual(H):
        M, D, _ = law(H)
        return H.reshape(-1) - N @ M.reshape(-1) - Hext.reshape(-1), D

    def times(X):
        return torch.einsum("rea,eab->reb", N4, X).reshape(3 * n, 3 * n)

    H = drive.reshape(n, 3)
    for _ in range(6):
        for _ in range(10):
            H = 0.5 * (H + torch.linalg.solve(eye - times(law(H)[2]), drive).reshape(n, 3))
        r, D = residual(H)
        for _ in range(40):
            dH = torch.linalg.solve(eye - times(D), -r).reshape(n, 3)
            lam = 1.0
            while lam > 1e-3:
                r2, D2 = residual(H + lam * dH)
                if r2.norm() < r.norm():
                    break
                lam *= 0.5
            else:
                break
            H, r, D = H + lam * dH, r2, D2
        if float(r.norm()) < 1e-11 * float(drive.norm()):
            break
    return H, float(r.norm() / drive.norm())


def _dipole_field(blocks, coil, m):
    E = _elements(blocks)
    c, d, m = _t(E["c"]), _t(E["d"]), _t(m)
    return lambda q: _blocks_field(q, c, d, m, DIPOLE_IMAGES) + _coil_field(q, coil)


def _track(field, init, case):
    """Rows (y, x, x', z, z') of one classical Runge-Kutta step per interval."""
    Y = np.atleast_2d(init).astype(float)
    n, (y0, y1) = case["npts"], BEAM[1]
    step = (y1 - y0) / (n - 1)
    k = -2.99792458e5 / (1e9 * BEAM[0])   # charge over momentum, 1 / (T mm)

    def slope(y, F):
        x, xd, z, zd = F.T
        B = field(_t(np.stack([x, np.full_like(x, y), z], axis=1))).cpu().numpy()
        g = k * np.sqrt(1.0 + xd * xd + zd * zd)
        return np.stack([xd, -g * (zd * B[:, 1] - (1.0 + xd * xd) * B[:, 2] + xd * zd * B[:, 0]),
                         zd, g * (xd * B[:, 1] - (1.0 + zd * zd) * B[:, 0] + xd * zd * B[:, 2])], axis=1)

    out = np.zeros((len(Y), n, 5))
    y = y0
    for i in range(n):
        out[:, i, 0], out[:, i, 1:] = y, Y
        if i < n - 1:
            k1 = slope(y, Y)
            k2 = slope(y + 0.5 * step, Y + 0.5 * step * k1)
            k3 = slope(y + 0.5 * step, Y + 0.5 * step * k2)
            k4 = slope(y + step, Y + step * k3)
            Y = Y + step / 6.0 * (k1 + 2 * k2 + 2 * k3 + k4)
            y += step
    return out[0] if case["ntraj"] == 1 else out


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "field_magnets":
            blocks, P = _magnets(case, seed)
            E = _elements(blocks)
            c, d, m = _t(E["c"]), _t(E["d"]), _t(E["mr"])
            B = _chunked(lambda q: _blocks_field(q, c, d, m, [((1, 1, 1), 1.0)]), _t(P), len(c)).cpu().numpy()
            return B[0] if case["npts"] == 1 else B
        if kind == "field_dipole":
            blocks, coil, rng = _dipole(case, seed)
            f = _dipole_field(blocks, coil, _yoke_m(blocks, seed))
            return _chunked(f, _t(_grid_in_gap(case["npts"], rng)), len(_elements(blocks)["c"])).cpu().numpy()
        if kind == "trajectory":
            blocks, coil, rng = _dipole(case, seed)
            return _positions_and_angles(_track(_dipole_field(blocks, coil, _yoke_m(blocks, seed)), _beam(case, rng), case))
        if kind == "field_tets":
            V, m, P = _tets(case, seed)
            V, m = _t(V), _t(m)
            terms = _tet_terms(V)
            return _chunked(lambda q: _tets_field(q, V, m, terms), _t(P), len(V)).cpu().numpy()
        if kind == "solve_tets":
            if case["ntets"] > 4500:
                return None
            V = _t(_tets(case, seed)[0])
            N = _tets_matrix(V, _tet_terms(V))
            n3 = N.shape[0]
            h = _t(_background(seed)).repeat(n3 // 3)
            A = torch.eye(n3, dtype=N.dtype, device=N.device) - 1000.0 * N
            mr = _t([0.0, 0.0, 1e-12]).repeat(n3 // 3)
            return torch.linalg.solve(A, 1000.0 * h + mr).reshape(-1, 3).cpu().numpy()
        if kind in ("solve_magnets", "solve_dipole"):
            if kind == "solve_magnets":
                E = _elements(_magnets(case, seed)[0])
                images, coil = [((1, 1, 1), 1.0)], None
            else:
                blocks, coil, _ = _dipole(case, seed)
                E, images = _elements(blocks), DIPOLE_IMAGES
            c = _t(E["c"])
            N = _matrix_rows(c, c, _t(E["d"]), images)
            Hext = torch.zeros_like(c) if coil is None else _coil_field(c, coil)
            return _relaxed_m(E, N, Hext)
        if kind == "grad_hybrid":
            if case["npairs"] * (case["pole"] ** 3 + 12) > 1600:
                return None
            blocks, P, _ = _hybrid(case, seed)
            E = _elements(blocks)
            c, d = _t(E["c"]), _t(E["d"])
            M = _relaxed_m(E, _matrix_rows(c, c, d, HYBRID_IMAGES), torch.zeros_like(c))
            if M is None:
                return None
            F = _chunked(lambda q: _blocks_field(q, c, d, _t(M), HYBRID_IMAGES), _t(P), len(c)).cpu().numpy()
            return dict(F=F, M=M, mr=None, chi=None, centre=None, dims=None)
    return _exact_gradient(case, seed)


def _matrix_rows(P, c, d, images):
    step = max(1, int(3e6 // len(c)))
    return torch.cat([_blocks_matrix(P[i:i + step], c, d, images) for i in range(0, len(P), step)])


def _relaxed_m(E, N, Hext):
    law, chi, Mr = _law(E["mats"], E["mr"])
    if all(m[0] == "lin" for m in E["mats"]):
        n = len(E["mats"])
        X = torch.block_diag(*chi)
        A = torch.eye(3 * n, dtype=N.dtype, device=N.device) - X @ N
        return torch.linalg.solve(A, X @ Hext.reshape(-1) + Mr.reshape(-1)).reshape(-1, 3).cpu().numpy()
    H, rel = _relax(N, Hext, law, Mr)
    return law(H)[0].cpu().numpy() if rel < 1e-11 else None


def _exact_gradient(case, seed):
    """F, M and the gradients of sum(W F) of the linear undulator, by autograd."""
    blocks, P, W = _undulator(case, seed)
    E = _elements(blocks)
    one = [((1, 1, 1), 1.0)]
    n = len(E["c"])
    if n * (n + len(P)) > 6e6:
        return None
    _, chi, _ = _law(E["mats"], E["mr"])
    c, d, mr, chi = (x.clone().requires_grad_(True) for x in (_t(E["c"]), _t(E["d"]), _t(E["mr"]), chi))
    N = _blocks_matrix(c, c, d, one).reshape(3 * n, n, 3)
    A = torch.eye(3 * n, dtype=torch.float64, device=DEV).reshape(n, 3, 3 * n) \
        - torch.einsum("eab,ebk->eak", chi, N.reshape(n, 3, 3 * n))
    M = torch.linalg.solve(A.reshape(3 * n, 3 * n), mr.reshape(-1))
    F = (_blocks_matrix(_t(P), c, d, one) @ M).reshape(-1, 3)
    (F * _t(W)).sum().backward()
    out = dict(F=F, M=M.reshape(-1, 3), mr=mr.grad, chi=chi.grad, centre=c.grad, dims=d.grad)
    return {k: v.detach().cpu().numpy() for k, v in out.items()}
