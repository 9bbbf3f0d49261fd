"""The far-field series (kemcu_series.cuh, compiled here as plain C++) against the element integrals of
the C restatement of the reference: wherever a tier may be taken (at its cut and beyond, every
direction), triangles of any shape, rectangles of any aspect, skew parallelograms and wires."""

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from kassiopeia_b200 import geometry as G
from oracle import port

HERE = os.path.dirname(os.path.abspath(__file__))
DP = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def series(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("series") / "series_host.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", so, os.path.join(HERE, "cxx", "series_host.cc")],
                   check=True)
    lib = C.CDLL(so)
    x, w = np.polynomial.legendre.leggauss(7)
    gx, gw = np.ascontiguousarray(.5 + .5 * x), np.ascontiguousarray(.5 * w)

    def run(rec, general, mixed, tier, P):
        P = np.ascontiguousarray(P)
        out, cuts = np.zeros((len(P), 4)), np.zeros(3)
        lib.series_host(*(a.ctypes.data_as(DP) if isinstance(a, np.ndarray) else a
                          for a in (rec, general, mixed, tier, gx, gw, len(P), P, out, cuts)))
        return out, cuts
    return run


SHAPES = {  # sides in the plane, general form
    "square": (G.RECTANGLE, [1., 0], [0, 1.], 0), "3:1": (G.RECTANGLE, [.06, 0], [0, .02], 0),
    "1:50": (G.RECTANGLE, [.02, 0], [0, 1.], 0), "wire": (G.LINE_SEGMENT, [.3, 0], [0, 0], 0),
    "equilateral": (G.TRIANGLE, [1., 0], [.5, .8660254037844386], 1), "right": (G.TRIANGLE, [.1, 0], [0, .1], 1),
    "sliver": (G.TRIANGLE, [1., 0], [.95, .03], 1), "obtuse": (G.TRIANGLE, [1., 0], [-.7, .2], 1),
    "rectangle in a general tile": (G.RECTANGLE, [1., 0], [0, .4], 1), "skew": (G.RECTANGLE, [1., 0], [.6, .8], 1),
}


@pytest.mark.parametrize("name", SHAPES)
@pytest.mark.parametrize("mixed", [0, 1])
def test_series_is_the_rules_sum_beyond_its_cuts(series, name, mixed):
    shape, a, b, general = SHAPES[name]
    rng = np.random.default_rng(len(name) + mixed)
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    a, b, p0 = q[:, :2] @ np.array(a, float), q[:, :2] @ np.array(b, float), rng.normal(size=3) * .3
    if shape == G.LINE_SEGMENT:
        m = G.line_segments(p0[None], (p0 + a)[None], 1e-4, 1.)
    elif shape == G.TRIANGLE:
        m = G.triangles_from_vertices(p0[None], (p0 + a)[None], (p0 + b)[None], 1.)
    else:
        m = G.rectangles_from_corners(p0[None], (p0 + a)[None], (p0 + b)[None], 1.)
    A, B = np.linalg.norm(a), np.linalg.norm(b)
    rec = np.zeros(32)
    f = 1 / 3 if shape == G.TRIANGLE else .5
    rec[0], rec[11:14], rec[14:17], rec[17:20], rec[25] = A, a, b, p0 + f * (a + b), shape
    size = (A + B + np.linalg.norm(b - a)) / 3 if shape == G.TRIANGLE else .5 * (A + B) if shape == G.RECTANGLE else A
    k = 1. / (4 * np.pi * 8.8541878128e-12)
    area = .5 * np.linalg.norm(np.cross(a, b)) if shape == G.TRIANGLE else A * B  # a rectangle's sides, as the record
    rec[24] = area * k if shape != G.LINE_SEGMENT else np.pi * 1e-4 * k  # a wire's record holds it per length
    cut0 = {G.TRIANGLE: 3.42, G.RECTANGLE: 4.6, G.LINE_SEGMENT: 2.}[shape]
    rec[29] = (cut0 * size) ** 2
    oracle = port.PortProblem(m)
    _, cuts = series(rec, general, mixed, 3, np.zeros((2, 3)))
    assert cuts[0] >= cuts[1] >= cuts[2] > 1.4 * cut0 * size  # nested, and never at an analytic pair
    u = rng.normal(size=(60, 3))
    u[:8], u[8:16], u[16:24] = a, -b if shape != G.LINE_SEGMENT else a, q[:, 2]
    u /= np.linalg.norm(u, axis=1)[:, None]
    for tier in (3, 2, 1):
        for far in (1.0000001, 1.3, 4., 1000.):
            P = rec[17:20] + far * cuts[3 - tier] * u
            out, _ = series(rec, general, mixed, tier, P)
            want = oracle.element_field(0, P)
            # FP64: rounding of a 33-node sum and of the series' ~60 operations, the first orders left out and the FP32
            # tail a few 1e-15 of the field in the worst direction at a cut; also the rule's own defect
            # from the exact integral, below 1e-14 at the cuts of slender elements. MIXED: 1e-14 for the
            # orders left out and 4e-7 of the first order in FP32, which the cuts hold to 3e-13
            tol = 3e-14 if not mixed else 5e-13
            err = np.linalg.norm(out[:, :3] - want[:, :3], axis=1) / np.linalg.norm(want[:, :3], axis=1)
            assert err.max() <= tol and np.abs(out[:, 3] / want[:, 3] - 1).max() <= tol, (tier, far, err.max())


@pytest.mark.parametrize("aspect", [1., .95, .84, .8, .5, .1])
def test_half_of_the_mixed_cuts_is_outside_the_analytic_band(series, aspect):
    # the FP32 form takes the series from there on, and its analytic pairs are FP64
    for shape, b in ((G.RECTANGLE, [0., aspect]), (G.RECTANGLE, [.3 * aspect, .9 * aspect]), (G.TRIANGLE, [.5, aspect])):
        A, B = 1., np.linalg.norm(b)
        rec = np.zeros(32)
        rec[0], rec[11], rec[14:16], rec[25] = A, 1., b, shape
        size = (A + B + np.hypot(1. - b[0], b[1])) / 3 if shape == G.TRIANGLE else .5 * (A + B)
        rec[29] = ({G.TRIANGLE: 3.42, G.RECTANGLE: 4.6}[shape] * size) ** 2
        _, cuts = series(rec, int(shape == G.TRIANGLE or b[0] != 0.), 1, 3, np.zeros((2, 3)))
        assert .5 * cuts.min() > np.sqrt(rec[29])
