"""The analytic near field from the near records (rwg_pair), through the fast multipole field solver whose
direct pairs are all analytic: points at every kind of distance from triangles and rectangles (off and
almost in the plane, over edges and corners, on edge lines, at vertices, in the plane inside and
outside), against the C restatement's analytic integrals, which those points take at this distance."""

import numpy as np
import pytest

import kassiopeia_b200 as K
from kassiopeia_b200 import geometry as G
from oracle import port

pytestmark = pytest.mark.gpu

P0, A, B = np.array([.1, -.2, .3]), np.array([.3, .1, 0.]), np.array([-.05, .15, .2])


@pytest.mark.parametrize("shape", ["triangle", "rectangle", "sliver"])
def test_near_points(shape):
    b = B - (B @ A) / (A @ A) * A
    if shape == "rectangle":
        m = G.rectangles_from_corners([P0], [P0 + A], [P0 + b], 1.)
    else:
        b = B if shape == "triangle" else A * .9 + .01 * b
        m = G.triangles_from_vertices([P0], [P0 + A], [P0 + b], 1.)
    n = np.cross(A, b)
    n /= np.linalg.norm(n)
    size = np.linalg.norm(A)
    base = [P0 + s * A + t * b for s, t in ((.3, .2), (.5, 0.), (0., .5), (.5, .5), (0., 0.), (1., 0.), (0., 1.), (1.2, .3),
                                            (-.4, 0.), (2., 0.), (-.3, -.5), (.05, .04))]
    hs = [.5, .1, 1e-2, 1e-4, 3e-8, 1e-8, 0., -1e-7, -1e-3, -.3]
    P = np.array([p + h * size * n for p in base for h in hs])
    o = port.PortProblem(m)
    o.set_sigma(np.array([1e-9]))
    want = o.field(P)
    ok = np.isfinite(want).all(1)
    with K.CUDAElectrostaticContext(0) as ctx:
        ctx.SetGeometry(m)
        ctx.SetSigma(np.array([1e-9]))
        ctx.ConfigureFFTM(degree=2, maximum_tree_depth=1, world_center=[0., 0., 0.], world_length=8., top_level_divisions=2)
        got = ctx.FFTMField(P[ok])
        # An edge's logarithm has the argument R + s, s the way along its line: at a distance h from the line
        # and s < 0 that is h^2 / 2R with an absolute rounding error of eps R, so the value carries
        # 2 eps (R / h)^2 of each of its three or four edges, in this code and in the restatement alike (and
        # on a line itself, nothing is left to compare). The solid angle at a distance z from the plane is 2 pi
        # less angles of the size of z / R, each of arccosines or a product of complex numbers near the real
        # axis: eps R / z per edge. In the plane itself the field jumps across the element and the rounding of
        # the point's distance decides the side: the potential is compared. Elsewhere some tens of roundings.
        v = [P0, P0 + A, P0 + A + b, P0 + b] if shape == "rectangle" else [P0, P0 + A, P0 + b]
        h = np.array([[np.linalg.norm(np.cross(p - v[k], v[k - 1] - v[k])) / np.linalg.norm(v[k - 1] - v[k])
                       for k in range(len(v))] for p in P[ok]]).min(1)
        R = np.array([[np.linalg.norm(p - q) for q in v] for p in P[ok]]).max(1)
        line = h < 1e-9 * size
        z = np.abs(np.tile(hs, len(base)))[ok] * size
        tol = 1e-12 + 2.2e-16 * len(v) * (2 * (R / np.where(line, 1., h)) ** 2 + R / np.where(z > 0., z, np.inf))
        err = np.abs(got - want[ok]) / np.abs(want[ok])[~line].max(0)
        err[z == 0., :3] = 0.
        assert np.all((err <= tol[:, None])[~line]), (err.max(1) / tol)[~line].max()
