"""The work that programs have this framework do, as timed cases.

Every case is one call (or the short run of calls) of a user's program through the public Python
entry points of :mod:`kassiopeia_b200`: field maps by the direct sum, products with the
boundary-integral operator (matrix-free and assembled), charge-density solves (GMRES from the
geometry on, Robin Hood), RK8 tracking, the adjoint, the fast multipole field and product, and the
axisymmetric direct sum. Sizes are those of the repository's configurations and tests, from a
single probe point to the 44,000-element coax.

``exact`` restates the element integrals (cubature bands, analytic near field, wires, conic
sections) in plain torch, in 64 bits.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import kassiopeia_b200 as K
from kassiopeia_b200 import geometry as G

PRECISION = {"fp64": K.FP64, "mixed": K.MIXED, "fp32": K.FP32}
WHAT = {"both": K.FIELD_AND_POTENTIAL, "potential": K.POTENTIAL, "field": K.FIELD}
MODE = {"plain": K.SOLVE_PLAIN, "mixed": K.SOLVE_MIXED, "assembled": K.SOLVE_ASSEMBLED,
        "assembled64": K.SOLVE_ASSEMBLED_FP64, "fp32": K.SOLVE_FP32}


# ------------------------------------------------------------------------------------- cases
def listed():
    return [
        # one probe: what a program that asks for the field point by point pays (latency)
        dict(name="field-probe", kind="field", mesh="sphere", scale=3, points=1, precision="fp64", what="both",
             device=False),
        # an ordinary field map with wires: a box of rectangles refined to its edges, a wire grid
        # inside, host arrays, points in caller order, a ragged count
        dict(name="field-map", kind="field", mesh="cage", scale=24, points=10007, precision="fp64", what="both",
             device=False),
        # the large direct sum: the 44,000-element coax, device arrays, the MIXED form
        dict(name="field-large", kind="field", mesh="coax", scale=100, points=400000, precision="mixed", what="both",
             device=True),
        # the matrix-free product, once per iteration of the plain solves (triangles, one column)
        dict(name="matvec-free", kind="matvec", mesh="rings", scale=60, rhs=1, precision="fp64", assembled=False),
        # the product with the operator kept in device memory, eight columns at once
        dict(name="matvec-assembled", kind="matvec", mesh="coax", scale=80, rhs=8, precision="fp64", assembled=True),
        # from a new geometry to its charge densities: records, assembly, GMRES, refinement
        dict(name="solve-new-geometry", kind="solve", mesh="coax", scale=52, rhs=1, mode="assembled", tol=1e-10),
        # Robin Hood on the 1,280-triangle sphere, columns computed on the fly
        dict(name="robin-hood", kind="robinhood", mesh="sphere", scale=3, assembled=False, tol=1e-8),
        # electrons in the field of the sphere, all tracks a few steps
        dict(name="track", kind="track", mesh="sphere", scale=3, tracks=16384, steps=4, precision="mixed"),
        # the adjoint of a field map: gradients to densities and vertices
        dict(name="adjoint", kind="adjoint", mesh="sphere", scale=5, points=4096, precision="fp64"),
        # the fast multipole field map of a million points
        dict(name="fftm-field", kind="fftm-field", mesh="coax", scale=100, points=1000000, degree=8, depth=6,
             what="both"),
        # the fast multipole product, once per iteration of its solves
        dict(name="fftm-matvec", kind="fftm-matvec", mesh="coax", scale=100, rhs=1, degree=8, depth=5),
        # conic sections and rings, device arrays
        dict(name="axisym-field", kind="axisym", scale=800, points=20015, what="both"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _points(rng, lo, hi):
    """A count of points over [lo, hi], ragged above a thousand (the last warp and block part full)."""
    n = _log(rng, lo, hi)
    return n if n < 1024 else n // 64 * 64 - rng.randint(1, 19)


def _mesh_choice(rng, most):
    while True:
        mesh = rng.choice(["sphere", "coax", "rings", "cage"])
        scale = rng.randint(1, 5) if mesh == "sphere" else _log(rng, 6, 100) if mesh != "cage" else _log(rng, 3, 60)
        if mesh_size(mesh, scale) <= most:
            return mesh, scale


def draw(rng):
    kind = rng.choice(["field", "field", "field", "matvec", "matvec", "solve", "robinhood", "track", "adjoint",
                       "fftm-field", "fftm-matvec", "axisym"])
    if kind == "field":
        mesh, scale = _mesh_choice(rng, 44000)
        points = _points(rng, 1, min(400000, int(1.1e10 / mesh_size(mesh, scale))))
        return dict(kind=kind, mesh=mesh, scale=scale, points=points, precision=rng.choice(["fp64", "mixed", "fp32"]),
                    what=rng.choice(["both", "both", "potential", "field"]), device=points > 50000 or rng.random() < .3)
    if kind == "matvec":
        mesh, scale = _mesh_choice(rng, 30000)
        return dict(kind=kind, mesh=mesh, scale=scale, rhs=rng.choice([1, 1, 2, 5, 8]),
                    precision=rng.choice(["fp64", "mixed", "fp32"]), assembled=rng.random() < .5)
    if kind == "solve":
        mesh, scale = _mesh_choice(rng, 12000)
        return dict(kind=kind, mesh=mesh, scale=scale, rhs=rng.choice([1, 1, 3, 8]), mode=rng.choice(sorted(MODE)),
                    tol=rng.choice([1e-8, 1e-10]))
    if kind == "robinhood":
        return dict(kind=kind, mesh="sphere", scale=rng.choice([1, 2, 3]), assembled=rng.random() < .5,
                    tol=rng.choice([1e-6, 1e-8]))
    if kind == "track":
        mesh, scale = "sphere", rng.randint(1, 4)
        steps = rng.randint(1, 6)
        tracks = _log(rng, 33, min(20000, int(8e7 / (steps * mesh_size(mesh, scale)))))
        return dict(kind=kind, mesh=mesh, scale=scale, tracks=tracks, steps=steps,
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "adjoint":
        return dict(kind=kind, mesh="sphere", scale=rng.choice([4, 5]), points=_points(rng, 20, 4096),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "fftm-field":
        return dict(kind=kind, mesh=rng.choice(["coax", "rings"]), scale=_log(rng, 25, 100),
                    points=_points(rng, 1000, 1000000), degree=rng.randint(3, 10), depth=rng.choice([4, 5, 6]),
                    what=rng.choice(["both", "both", "potential", "field"]))
    if kind == "fftm-matvec":
        return dict(kind=kind, mesh=rng.choice(["coax", "rings"]), scale=_log(rng, 25, 100),
                    rhs=rng.choice([1, 1, 3, 8]), degree=rng.randint(2, 10), depth=rng.choice([4, 5]))
    return dict(kind=kind, scale=_log(rng, 40, 800), points=_points(rng, 1, 20000),
                what=rng.choice(["both", "potential", "field"]))


# ------------------------------------------------------------------------------------- meshes
def mesh_size(mesh, scale):
    if mesh == "sphere":
        return 20 * 4 ** scale
    if mesh == "coax":  # two cylinders of scale x 2 scale rectangles, 4 x 10 scale cap triangles
        return 4 * scale * scale + 40 * scale
    if mesh == "rings":
        return 8 * 2 * scale * max(2, scale // 2)
    return 6 * scale * scale + 9 * scale  # cage


def make_mesh(mesh, scale, seed):
    if mesh == "sphere":
        return G.icosphere(scale)
    if mesh == "coax":
        return G.coax(n_phi=scale, n_z=2 * scale)
    if mesh == "rings":
        return G.stacked_rings(n_rings=8, n_phi=scale, n_z=max(2, scale // 2), seed=seed)
    box = G.cube(scale)
    i, j = np.meshgrid(np.arange(9), np.arange(scale), indexing="ij")
    x, z = -.4 + .1 * i.ravel(), -.4 + .8 * j.ravel() / scale
    p0 = np.stack([x, 0 * x + .13, z], axis=1)
    wires = G.line_segments(p0, p0 + np.array([0., 0., .8 / scale]), 2e-4, -1.)
    return box.concat(wires)


def make_points(mesh, n, seed):
    if mesh == "coax":
        return G.gap_points(n, seed=seed)
    if mesh == "sphere":
        return G.shell_points(n, seed=seed)
    return np.random.default_rng(seed).uniform(-1.2, 1.2, (n, 3))


def make_points_axisym(n, seed):
    """Points of the gap off the electrodes and the wire rings at its middle."""
    P = G.gap_points(2 * n + 50, r_in=.51, r_out=.99, length=3.98, seed=seed)
    return P[np.abs(np.hypot(P[:, 0], P[:, 1]) - .75) > .002][:n].copy()


def make_sigma(m, seed):
    """Surface densities of the sizes and signs of a solved electrode system of +-1 kV."""
    rng = np.random.default_rng(seed + 1)
    return 1e-8 * np.sign(m.value + .5) * (1. + .2 * rng.normal(size=m.n))


def make_rhs(m, rhs, seed):
    """Potentials of the electrodes (the distinct boundary values) drawn per column, and a small
    position-dependent part (an external field)."""
    rng = np.random.default_rng(seed + 2)
    _, which = np.unique(m.value, return_inverse=True)
    b = rng.uniform(-1000., 1000., (rhs, which.max() + 1))[:, which]
    b = b + 50. * rng.normal(size=(rhs, 3)) @ m.centroids().T
    return b[0] if rhs == 1 else b


# ------------------------------------------------------------------------------------- passes
def prepare(case, seed):
    kind = case["kind"]
    if kind == "axisym":
        m = G.conic_coax(n_z=case["scale"], n_cap=max(2, case["scale"] // 10), n_rings=16)
    else:
        m = make_mesh(case["mesh"], case["scale"], seed)
    s = dict(case=case, mesh=m, ctx=K.CUDAElectrostaticContext(0))
    ctx = s["ctx"]
    if kind == "solve":
        if case["rhs"] == 1:  # the boundary values themselves
            m.value = make_rhs(m, 1, seed)
            s["b"] = None
        else:
            s["b"] = make_rhs(m, case["rhs"], seed)
        return s
    ctx.SetGeometry(m)
    if kind in ("field", "fftm-field", "axisym"):
        ctx.SetSigma(make_sigma(m, seed))
        if kind == "axisym":
            P = make_points_axisym(case["points"], seed)
        else:
            P = make_points(case["mesh"], case["points"], seed)
        s["P"] = P
        if kind == "fftm-field":
            ctx.ConfigureFFTM(degree=case["degree"], maximum_tree_depth=case["depth"])
        if kind != "field" or case["device"]:
            s["dP"] = torch.from_numpy(P).cuda()
            s["dO"] = torch.empty((len(P), 4), dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
    elif kind in ("matvec", "fftm-matvec"):
        s["x"] = np.stack([make_sigma(m, seed + 17 * r) for r in range(case["rhs"])])
        if case["rhs"] == 1:
            s["x"] = s["x"][0]
        if kind == "fftm-matvec":
            ctx.ConfigureFFTM(degree=case["degree"], maximum_tree_depth=case["depth"])
            ctx.FFTMMultiply(s["x"])  # the near part of the operator is kept from the first product
        elif case["assembled"]:
            ctx.Multiply(s["x"], precision=PRECISION[case["precision"]], assembled=True)
    elif kind == "robinhood":
        s["b"] = make_rhs(m, 1, seed)
        if case["assembled"]:
            ctx.Multiply(s["b"], assembled=True)
    elif kind == "track":
        ctx.SetSigma(make_sigma(m, seed) * 1e-3)
        s["state"] = G.electrons(case["tracks"], seed=seed)
    elif kind == "adjoint":
        ctx.SetSigma(make_sigma(m, seed))
        s["P"] = G.shell_points(case["points"], r_min=1.3, seed=seed)
        s["w"] = np.random.default_rng(seed + 3).normal(size=(case["points"], 4))
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "field" and not case["device"]:
        return ctx.ElectricFieldAndPotential(s["P"], precision=PRECISION[case["precision"]], what=WHAT[case["what"]])
    if kind in ("field", "axisym"):
        ctx.FieldDevice(s["dP"].data_ptr(), len(s["P"]), s["dO"].data_ptr(),
                        precision=PRECISION[case.get("precision", "fp64")], what=WHAT[case["what"]])
        return s["dO"]
    if kind == "fftm-field":
        ctx.FFTMFieldDevice(s["dP"].data_ptr(), len(s["P"]), s["dO"].data_ptr(), what=WHAT[case["what"]])
        return s["dO"]
    if kind == "matvec":
        return ctx.Multiply(s["x"], precision=PRECISION[case["precision"]], assembled=case["assembled"])
    if kind == "fftm-matvec":
        return ctx.FFTMMultiply(s["x"])
    if kind == "solve":
        ctx.SetGeometry(s["mesh"])
        x, _ = ctx.Solve(s["b"], tol=case["tol"], max_iter=400, mode=MODE[case["mode"]])
        return x
    if kind == "robinhood":
        x, _ = ctx.SolveRobinHood(s["b"], tol=case["tol"], assembled=case["assembled"])
        return x
    if kind == "track":
        st, steps, status, _ = ctx.TrackRK8(s["state"], 1e-11, 10000, step_budget=case["steps"], sphere_radius=1.0,
                                            precision=PRECISION[case["precision"]])
        return {"state": st, "steps": steps, "status": status}
    ds, dv = ctx.FieldVJP(s["P"], s["w"], precision=PRECISION[case["precision"]])
    return {"dsigma": ds, "dvertices": dv}


# ------------------------------------------------------------------------------------- floors
# One element-point pair of the direct sum at its least: the distance (8 operations), its inverse
# square root (8), the two leading corrections of the element's extent (14), the sums into four
# outputs (10) or one.
FLOP_BOTH, FLOP_POT = 40., 25.


def work(case):
    kind = case["kind"]
    if kind == "axisym":
        n = 2 * case["scale"] + 2 * max(2, case["scale"] // 10) + 16
        p = case["points"]  # 21 nodes on a conic section, K and E of each from series of ten terms
        return {"bytes": 80. * n + 56. * p, "flops": 21. * 90. * n * p}
    n = mesh_size(case["mesh"], case["scale"])
    if kind == "field":
        p = case["points"]
        return {"bytes": 96. * n + 56. * p, "flops": (FLOP_POT if case["what"] == "potential" else FLOP_BOTH) * n * p}
    if kind == "matvec" and not case["assembled"]:
        return {"bytes": 96. * n + 16. * n * case["rhs"], "flops": (FLOP_POT + 2. * case["rhs"]) * n * n}
    if kind == "matvec":
        size = 8. if case["precision"] == "fp64" else 4.
        return {"bytes": size * n * n + 16. * n * case["rhs"], "flops": 2. * n * n * case["rhs"]}
    if kind == "solve":  # the operator once, then ~60 products with it (its FP32 copy at the least)
        return {"bytes": 12. * n * n + 60. * 4. * n * n, "flops": (FLOP_POT + 120. * case["rhs"]) * n * n}
    if kind == "robinhood":  # ~12 n corrections of one column each
        return {"bytes": 12. * n * n * 8. if case["assembled"] else 96. * n, "flops": 12. * n * n * FLOP_POT}
    if kind == "track":
        return {"bytes": 96. * n + 136. * case["tracks"], "flops": 12. * FLOP_BOTH * n * case["tracks"] * case["steps"]}
    if kind == "adjoint":
        return {"bytes": 176. * n + 56. * case["points"], "flops": 2. * FLOP_BOTH * n * case["points"]}
    terms = (case["degree"] + 1.) ** 2
    if kind == "fftm-field":
        return {"bytes": 96. * n + 56. * case["points"], "flops": (30. * terms + 300.) * case["points"]}
    return {"bytes": 100. * n + 16. * n * case["rhs"], "flops": (30. * terms + 300.) * n * case["rhs"]}


def tolerance(case):
    kind = case["kind"]
    low = case.get("precision")
    if kind in ("field", "matvec"):
        if low == "fp32":  # 32-bit far field (or 32-bit operator entries)
            return {"rel": 1e-6, "max": 1e-5}
        if low == "mixed" and case.get("assembled"):
            return {"rel": 1e-6, "max": 1e-5}
        # MIXED: one Newton step on a 2^-22 estimate, 1e-13 a term; "max" for values near zero
        return {"rel": 2e-12, "max": 1e-9} if low == "mixed" else {"rel": 1e-13, "max": 1e-10}
    if kind == "solve":  # a residual of tol and condition numbers of 30 to some hundreds
        return {"rel": 300. * case["tol"], "max": 1e5 * case["tol"]}
    if kind == "robinhood":  # the order of corrections follows the last bits; the residual does not
        return {"rel": 30. * case["tol"], "max": 1e3 * case["tol"]}
    if kind == "track":
        return {"rel": 1e-11, "max": 1e-8}
    if kind == "adjoint":
        return {"rel": 2e-11, "max": 1e-8} if low == "mixed" else {"rel": 1e-12, "max": 1e-9}
    if kind == "axisym":
        return {"rel": 1e-12, "max": 1e-9}
    return {"rel": 1e-11, "max": 1e-8}  # fast multipole sums, 64 bits


# ------------------------------------------------------------------------------------- exact
MOST_PAIRS = 1.5e9  # pairs that exact evaluates within its time
PI = math.pi
EPS0 = 8.8541878128e-12
FOURPI = 1. / (4. * PI * EPS0)


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _tri(orbits):
    """(s, t, w) of a triangle rule from its orbits (kind, alpha, beta, weight)."""
    out = []
    perms = {1: [(0, 1, 2)], 3: [(0, 1, 2), (1, 0, 2), (2, 1, 0)], -3: [(0, 1, 2), (1, 2, 0), (2, 0, 1)],
             6: [(0, 1, 2), (1, 0, 2), (2, 1, 0), (0, 2, 1), (2, 0, 1), (1, 2, 0)]}
    for kind, a, b, w in orbits:
        v = (a, b, 1. - a - b)
        out += [(v[p[1]], v[p[2]], w) for p in perms[kind]]
    return out


def _rules():
    """The numeric policy's cubature rules: {(shape, band): [(s, t, w)]}, node = P0 + s A N1 + t B N2.
    Triangles: Radon 7, Gatermann 12, Papanicolopulos 33; rectangles: Stroud C2 5-1, Tyler 12,
    Cools-Haegemans 33 points."""
    c, q = 1. / 3., math.sqrt(15.)
    r7, s7 = (1. + q) / 7., (1. - q) / 7.
    t7 = _tri([(1, c, c, 9. / 40.), (3, c + 2. * c * s7, c - c * s7, (155. + q) / 1200.),
               (3, c + 2. * c * r7, c - c * r7, (155. - q) / 1200.)])
    t12 = _tri([(-3, 0.6238226509439084e-1, 0.6751786707392436e-1, 2. * 0.2651702815743450e-1),
                (-3, 0.5522545665692000e-1, 0.3215024938520156, 2. * 0.4388140871444811e-1),
                (-3, 0.3432430294509488e-1, 0.6609491961867980, 2. * 0.2877504278497528e-1),
                (-3, 0.5158423343536001, 0.2777161669764050, 2. * 0.6749318700980879e-1)])
    t33 = _tri([(3, 4.570749859701478e-01, 2.714625070149261e-01, 6.254121319590276e-02),
                (3, 1.197767026828138e-01, 4.401116486585931e-01, 4.991833492806094e-02),
                (3, 2.359249810891690e-02, 4.882037509455416e-01, 2.426683808145203e-02),
                (3, 7.814843446812914e-01, 1.092578276593543e-01, 2.848605206887754e-02),
                (3, 9.507072731273288e-01, 2.464636343633559e-02, 7.931642509973638e-03),
                (6, 1.162960196779266e-01, 2.554542286385173e-01, 4.322736365941421e-02),
                (6, 2.303415635526714e-02, 2.916556797383410e-01, 2.178358503860756e-02),
                (6, 2.138249025617059e-02, 1.272797172335894e-01, 1.508367757651144e-02)])
    r, s, t = math.sqrt(.6), math.sqrt(1. / 3.), math.sqrt(14. / 15.)
    x7 = [(0, 0, 2. / 7.), (0, t, 5. / 63.), (0, -t, 5. / 63.)] + [(a * r, b * s, 5. / 36.) for a in (1, -1) for b in (1, -1)]
    w = math.sqrt(583.)
    r, s, t = math.sqrt(6. / 7.), math.sqrt((114. - 3. * w) / 287.), math.sqrt((114. + 3. * w) / 287.)
    x12 = [(r, 0, 49. / 810.), (-r, 0, 49. / 810.), (0, r, 49. / 810.), (0, -r, 49. / 810.)]
    x12 += [(a * s, b * s, (178981. + 2769. * w) / 1888920.) for a in (1, -1) for b in (1, -1)]
    x12 += [(a * t, b * t, (178981. - 2769. * w) / 1888920.) for a in (1, -1) for b in (1, -1)]
    X = [0.77880971155441942252, 0.95729769978630736566, 0.13818345986246535375, 0.94132722587292523695,
         0.47580862521827590507, 0.75580535657208143627, 0.69625007849174941396, 0.34271655604040678941]
    Y = [0.98348668243987226379, 0.85955600564163892859, 0.95892517028753485754, 0.39073621612946100068,
         0.85007667369974857597, 0.64782163718701073204, 0.70741508996444936217e-1, 0.40930456169403884330]
    W = [0.29991838864499131666e-1, 0.38174421317083669640e-1, 0.60424923817749980681e-1, 0.77492738533105339358e-1,
         0.11884466730059560108, 0.12976355037000271129, 0.21334158145718938943, 0.25687074948196783651]
    x33 = [(0., 0., 0.30038211543122536139 / 4.)]
    for a, b, v in zip(X, Y, W):
        x33 += [(a, b, v / 4.), (-a, -b, v / 4.), (-b, a, v / 4.), (b, -a, v / 4.)]
    half = lambda x: [(.5 + .5 * a, .5 + .5 * b, v) for a, b, v in x]  # noqa: E731
    return {(0, 1): t33, (0, 2): t12, (0, 3): t7, (1, 1): half(x33), (1, 2): half(x12), (1, 3): half(x7)}


CUTS = {0: (3.42, 30.4, 131.4), 1: (4.6, 44.6, 196.2), 2: (2., 27.7, 1e300)}


def _elements(m, V=None):
    """Element tensors; V: [n, 3, 3] vertices (P0, P1, P2) of triangles and rectangles to use instead."""
    dev = _dev()
    g = torch.tensor(np.asarray(m.geom), dtype=torch.float64, device=dev)
    shape = torch.tensor(np.asarray(m.shape), dtype=torch.int64, device=dev)
    line = (shape == 2)[:, None]
    if V is None:
        p0 = torch.where(line, g[:, 0:3], g[:, 2:5])
        a = torch.where(line, g[:, 3:6] - g[:, 0:3], g[:, 0:1] * g[:, 5:8])
        b = torch.where(line, torch.zeros_like(a), g[:, 1:2] * g[:, 8:11])
    else:
        p0, a, b = V[:, 0], V[:, 1] - V[:, 0], V[:, 2] - V[:, 0]
    A, B = a.norm(dim=1), b.norm(dim=1)
    tri = shape == 0
    f = (.5 - tri.double() / 6.)[:, None]
    size = torch.where(tri, (A + B + (b - a).norm(dim=1)) / 3., torch.where(line[:, 0], A, .5 * (A + B)))
    area = torch.linalg.cross(a, b).norm(dim=1)
    area = torch.where(tri, .5 * area, area)
    return dict(shape=shape, p0=p0, a=a, b=b, cen=p0 + f * a + f * b, size=size, pre=area * FOURPI, diam=g[:, 6])


def _cubature(E, j, P, nodes):
    d0, a, b = P - E["p0"][j], E["a"][j], E["b"][j]
    phi, fld = 0., 0.
    for s, t, w in nodes:
        d = d0 - s * a - t * b
        ir = (d * d).sum(1).rsqrt()
        phi = phi + w * ir
        fld = fld + (w * ir ** 3)[:, None] * d
    pre = E["pre"][j]
    return torch.cat([pre[:, None] * fld, (pre * phi)[:, None]], 1)


def _solid(u, v, w):
    x = 1. + (u * v).sum(1) + (u * w).sum(1) + (v * w).sum(1)
    return 2. * torch.atan2((u * torch.linalg.cross(v, w)).sum(1).abs(), x)


def _analytic(E, j, P, nv):
    """Potential and field of uniformly charged polygons (Rao-Wilton-Glisson), off their edges."""
    p0, a, b = E["p0"][j], E["a"][j], E["b"][j]
    v = [p0, p0 + a, p0 + b] if nv == 3 else [p0, p0 + a, p0 + a + b, p0 + b]
    n = torch.linalg.cross(a, b)
    n = n / n.norm(dim=1, keepdim=True)
    h = (n * (P - E["cen"][j])).sum(1)
    d = [x - P for x in v]
    r = [x.norm(dim=1) for x in d]
    il, iv = 0., 0.
    for i in range(nv):
        k = (i + 1) % nv
        u = v[k] - v[i]
        u = u / u.norm(dim=1, keepdim=True)
        sm, sp = (d[i] * u).sum(1), (d[k] * u).sum(1)
        up = r[i] + sm > r[k] - sp
        log = torch.where(up, torch.log((r[k] + sp) / (r[i] + sm)), torch.log((r[i] - sm) / (r[k] - sp)))
        m = torch.linalg.cross(u, n)
        il = il - (m * d[i]).sum(1) * log
        iv = iv + log[:, None] * m
    e = [x / y[:, None] for x, y in zip(d, r)]
    om = _solid(e[0], e[1], e[2])
    if nv == 4:
        om = om + _solid(e[2], e[3], e[0])
        q = P - p0
        s, t = (q * a).sum(1) / (a * a).sum(1), (q * b).sum(1) / (b * b).sum(1)
        inside = (s > 0) & (s < 1) & (t > 0) & (t < 1)
        om = torch.where(h.abs() < 1e-12, 2. * PI * inside.double(), om)
    else:
        om = torch.where((P - E["cen"][j]).norm(dim=1) <= 1e-12, 2. * PI, om)
    om = torch.where(h < 0, -om, om)
    return FOURPI * torch.cat([n * om[:, None] + iv, (-h * om - il)[:, None]], 1)


def _wire(E, j, P, band):
    p0, u, diam = E["p0"][j], E["a"][j], E["diam"][j]
    L = u.norm(dim=1)
    if band:
        x, w = np.polynomial.legendre.leggauss(16 if band == 1 else 4)
        phi, fld = 0., 0.
        for xi, wi in zip(x, w):
            d = P - p0 - (.5 + .5 * float(xi)) * u
            ir = (d * d).sum(1).rsqrt()
            phi = phi + .5 * float(wi) * L * ir
            fld = fld + (.5 * float(wi) * L * ir ** 3)[:, None] * d
        pre = .25 * diam / EPS0
        return torch.cat([pre[:, None] * fld, (pre * phi)[:, None]], 1)
    p1 = p0 + u
    Da, Db = (P - p0).norm(dim=1), (P - p1).norm(dim=1)
    t = ((P - p0) * u).sum(1) / L  # a point inside the wire: the potential on its surface
    rad = (P - p0 - (t / L)[:, None] * u).norm(dim=1)
    inside = (rad < .5 * diam) & (t >= -.5 * diam) & (t <= L + .5 * diam) & (Da + Db <= L + diam)
    Da = torch.where(inside, torch.sqrt(t * t + .25 * diam * diam), Da)
    Db = torch.where(inside, torch.sqrt((L - t) ** 2 + .25 * diam * diam), Db)
    phi = diam / (4. * EPS0) * torch.log((Da + Db + L) / (Da + Db - L))
    s = -2. * L * diam / (Da * (Da + Db + L) * (Da + Db - L) * Db * 4. * EPS0)
    return torch.cat([s[:, None] * (p1 * Da[:, None] - P * (Da + Db)[:, None] + p0 * Db[:, None]), phi[:, None]], 1)


RULES = _rules()


def _blocks(E, P, per):
    """(first point, pair point, pair element, values [pairs, 4]) over chunks of the points."""
    n = len(E["size"])
    step = max(1, int(per // n))
    for p0 in range(0, len(P), step):
        Q = P[p0:p0 + step]
        ratio = (Q[:, None, :] - E["cen"].detach()[None, :, :]).norm(dim=2) / E["size"].detach()
        for sh in (0, 1, 2):
            is_sh = (E["shape"] == sh)[None, :]
            if not bool(is_sh.any()):
                continue
            c = CUTS[sh]
            band = (ratio > c[0]).to(torch.int8) + (ratio > c[1]).to(torch.int8) + (ratio > c[2]).to(torch.int8)
            for bd in range(4):
                i, j = torch.nonzero(is_sh & (band == bd), as_tuple=True)
                for k in range(0, len(i), 1 << 22):
                    ii, jj = i[k:k + (1 << 22)], j[k:k + (1 << 22)]
                    if sh == 2:
                        v = _wire(E, jj, Q[ii], bd)
                    elif bd == 0:
                        v = _analytic(E, jj, Q[ii], 3 + sh)
                    else:
                        v = _cubature(E, jj, Q[ii], RULES[sh, bd])
                    yield p0, ii + p0, jj, v


def _field(E, sigma, P):
    out = torch.zeros((len(P), 4), dtype=torch.float64, device=P.device)
    for _, i, j, v in _blocks(E, P, 3e7):
        out.index_add_(0, i, v * sigma[j][:, None])
    return out


def _matrix(E):
    n = len(E["size"])
    A = torch.zeros((n, n), dtype=torch.float64, device=E["size"].device)
    for _, i, j, v in _blocks(E, E["cen"], 3e7):
        A[i, j] = v[:, 3]
    return A


# the 13-stage eighth-order scheme of the tracker (rows: stage values, last row: the step)
RK8 = [
    {0: 1 / 4}, {0: 5 / 72, 1: 1 / 72}, {0: 1 / 32, 2: 3 / 32}, {0: 106 / 125, 2: -408 / 125, 3: 352 / 125},
    {0: 1 / 48, 3: 8 / 33, 4: 125 / 528},
    {0: -1263 / 2401, 3: 39936 / 26411, 4: -64125 / 26411, 5: 5520 / 2401},
    {0: 37 / 392, 4: 1625 / 9408, 5: -2 / 15, 6: 61 / 6720},
    {0: 17176 / 25515, 3: -47104 / 25515, 4: 1325 / 504, 5: -41792 / 25515, 6: 20237 / 145800, 7: 4312 / 6075},
    {0: -23834 / 180075, 3: -77824 / 1980825, 4: -636635 / 633864, 5: 254048 / 300125, 6: -183 / 7000, 7: 8 / 11,
     8: -324 / 3773},
    {0: 12733 / 7600, 3: -20032 / 5225, 4: 456485 / 80256, 5: -42599 / 7125, 6: 339227 / 912000, 7: -1029 / 4180,
     8: 1701 / 1408, 9: 5145 / 2432},
    {0: -27061 / 204120, 3: 40448 / 280665, 4: -1353775 / 1197504, 5: 17662 / 25515, 6: -71687 / 1166400, 7: 98 / 225,
     8: 1 / 16, 9: 3773 / 11664},
    {0: 11203 / 8680, 3: -38144 / 11935, 4: 2354425 / 458304, 5: -84046 / 16275, 6: 673309 / 1636800, 7: 4704 / 8525,
     8: 9477 / 10912, 9: -1029 / 992, 11: 729 / 341},
    {0: 31 / 720, 5: 16 / 75, 6: 16807 / 79200, 7: 16807 / 79200, 8: 243 / 1760, 11: 243 / 1760, 12: 31 / 720},
]


def _track(E, sigma, state, dt, steps):
    q, mass, c2 = -G.ELEMENTARY_CHARGE, G.ELECTRON_MASS, G.SPEED_OF_LIGHT ** 2
    y = state.clone()
    n = len(y)
    count = np.zeros(n, np.int32)
    status = np.zeros(n, np.int32)
    active = torch.ones(n, dtype=torch.bool, device=y.device)
    for _ in range(steps):
        k = {}
        at = y[:, 2:8]
        for st in range(13):
            if st != 10:  # its derivative has no weight anywhere
                X = at if st == 0 else at + dt * sum(RK8[st - 1].get(i, 0.) * k[i] for i in k)
                gam = torch.sqrt(1. + (X[:, 3:] ** 2).sum(1) / (mass * mass * c2))
                k[st] = torch.cat([X[:, 3:] / (mass * gam)[:, None], q * _field(E, sigma, X[:, :3])[:, :3]], 1)
        w = RK8[12]
        new = y.clone()
        new[:, 0] += dt * sum(w.values())
        new[:, 1] += dt * sum(w[i] * k[i][:, :3].norm(dim=1) for i in w)
        new[:, 2:8] += dt * sum(w[i] * k[i] for i in w)
        y = torch.where(active[:, None], new, y)
        a = active.cpu().numpy()
        count[a] += 1
        hit = active & ((y[:, 2:5] ** 2).sum(1) <= 1.)
        status[hit.cpu().numpy()] = 1
        active = active & ~hit
    return {"state": y, "steps": count, "status": status}


def _ellip(k2):
    """K, E and (E - K) / k^2 by the arithmetic-geometric mean."""
    a, b = torch.ones_like(k2), torch.sqrt(1. - k2)
    s, t, f = torch.zeros_like(k2), torch.full_like(k2, .5), 1.  # s: sum 2^(n-1) c_n^2 / k^2 from n = 1
    for _ in range(8):
        c = .5 * (a - b)
        a, b = .5 * (a + b), torch.sqrt(a * b)
        s = s + f * c * c / k2.clamp_min(1e-300)
        f = 2. * f
    Kk = .5 * PI / a
    EK = -Kk * (t + s)
    return Kk, Kk + k2 * EK, EK


GLUECK = [0.2803440531305107, 1.648702325837748, -0.2027449845679092, 2.797927414021179, -0.9761199294532843,
          2.556499393738999, 0.1451083002645404, 1.311227127425048, 0.9324249063051143, 1.006631393098060]


def _axisym(m, sigma, P):
    """Conic sections and rings at points away from the generators (no subdivided near branch)."""
    dev = P.device
    g = torch.tensor(np.asarray(m.geom), dtype=torch.float64, device=dev)
    ring = torch.tensor(np.asarray(m.shape) == 4, device=dev)
    ra, za = g[:, 0], g[:, 1]
    rb, zb = torch.where(ring, ra, g[:, 2]), torch.where(ring, za, g[:, 3])
    L = torch.where(ring, torch.ones_like(ra), torch.hypot(ra - rb, za - zb))
    pre = 1. / (PI * EPS0) * torch.where(ring, 1. / (2. * PI * ra), torch.ones_like(ra))
    out = torch.zeros((len(P), 4), dtype=torch.float64, device=dev)
    step = max(1, int(4e6 // len(L)))
    for p0 in range(0, len(P), step):
        Q = P[p0:p0 + step]
        r, z = torch.hypot(Q[:, 0], Q[:, 1])[:, None], Q[:, 2:3]
        D = (torch.hypot(za - z, ra - r) + torch.hypot(zb - z, rb - r) - L).abs() / L
        acc = torch.zeros((3, len(Q), len(L)), dtype=torch.float64, device=dev)
        bands = [(ring[None, :].expand(len(Q), -1), 0), (~ring & (D >= 5e-2), 20),
                 (~ring & (D < 5e-2) & (D >= 5e-3), 100), (~ring & (D < 5e-3), 500)]
        for mask, n in bands:
            i, j = torch.nonzero(mask, as_tuple=True)
            if not len(i):
                continue
            rr, zz = r[i, 0], z[i, 0]
            tot = [0., 0., 0.]
            for k in range(n + 1):
                t = k / n if n else 0.
                w = 1. if not n else GLUECK[min(k, n - k)] if k < 10 or k > n - 10 else 1.
                R, dz = ra[j] + t * (rb[j] - ra[j]), zz - (za[j] + t * (zb[j] - za[j]))
                dr, s2 = rr - R, (R + rr) ** 2 + dz * dz
                eta, S = (dr * dr + dz * dz) / s2, torch.sqrt(s2)
                Kk, Ee, EK = _ellip((1. - eta).clamp_min(0.))
                tot[0] = tot[0] + w * R / S ** 3 * (-2. * R * EK + dr / eta * Ee)
                tot[1] = tot[1] + w * dz / S ** 3 * Ee / eta * R
                tot[2] = tot[2] + w * R * Kk / S
            f = pre[j] * (L[j] / n if n else 1.)
            for c in range(3):
                acc[c, i, j] = f * tot[c]
        er, ez, phi = (a @ sigma for a in acc)
        out[p0:p0 + step] = torch.stack([Q[:, 0] / r[:, 0] * er, Q[:, 1] / r[:, 0] * er, ez, phi], 1)
    return out


def _masked(out, what):
    if what == "potential":
        out[:, :3] = 0.
    elif what == "field":
        out[:, 3] = 0.
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("fftm-field", "fftm-matvec"):
        return None  # the expansions' truncation (1e-4) is part of the result and far above rounding
    dev = _dev()
    T = lambda x: torch.tensor(np.asarray(x), dtype=torch.float64, device=dev)  # noqa: E731
    if kind == "axisym":
        m = G.conic_coax(n_z=case["scale"], n_cap=max(2, case["scale"] // 10), n_rings=16)
        if m.n * case["points"] > 5e7:
            return None
        P = T(make_points_axisym(case["points"], seed))
        return _masked(_axisym(m, T(make_sigma(m, seed)), P), case["what"])
    m = make_mesh(case["mesh"], case["scale"], seed)
    pairs = float(m.n) * {"field": case.get("points", 0), "adjoint": 8 * case.get("points", 0),
                          "track": 12 * case.get("steps", 0) * case.get("tracks", 0)}.get(kind, m.n)
    if pairs > MOST_PAIRS:
        return None
    E = _elements(m)
    if kind == "field":
        return _masked(_field(E, T(make_sigma(m, seed)), T(make_points(case["mesh"], case["points"], seed))),
                       case["what"])
    if kind == "matvec":
        x = np.stack([make_sigma(m, seed + 17 * r) for r in range(case["rhs"])])
        y = torch.zeros((len(x), m.n), dtype=torch.float64, device=dev)
        X = T(x)
        for _, i, j, v in _blocks(E, E["cen"], 3e7):
            y.index_add_(1, i, v[:, 3] * X[:, j])
        return y[0] if case["rhs"] == 1 else y
    if kind in ("solve", "robinhood"):
        b = T(make_rhs(m, case.get("rhs", 1), seed))
        x = torch.linalg.solve(_matrix(E), b.reshape(-1, m.n).T).T
        return x[0] if case.get("rhs", 1) == 1 else x
    if kind == "track":
        return _track(E, T(make_sigma(m, seed) * 1e-3), T(G.electrons(case["tracks"], seed=seed)), 1e-11, case["steps"])
    # adjoint: the probes keep out of the analytic band, so a gradient is that of the rule's sum
    sigma, w = T(make_sigma(m, seed)), T(np.random.default_rng(seed + 3).normal(size=(case["points"], 4)))
    P = T(G.shell_points(case["points"], r_min=1.3, seed=seed))
    V = torch.stack([E["p0"], E["p0"] + E["a"], E["p0"] + E["b"]], 1).requires_grad_(True)
    ds = torch.zeros(m.n, dtype=torch.float64, device=dev)
    dv = torch.zeros((m.n, 9), dtype=torch.float64, device=dev)
    for p0 in range(0, len(P), 16):
        L = 0.
        for _, i, j, v in _blocks(_elements(m, V), P[p0:p0 + 16], 3e7):
            f = (v * w[p0 + i]).sum(1)
            ds.index_add_(0, j, f.detach())
            L = L + (f * sigma[j]).sum()
        dv += torch.autograd.grad(L, V)[0].reshape(m.n, 9)
    return {"dsigma": ds, "dvertices": dv}
