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
    # 1e-6 of an edge or plane the integrals' own terms cancel by as much: the tolerance is in units of the
    # largest value, and within 1e-6 of an edge line the logarithm's argument carries 1e-10
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
        assert np.all(np.abs(got - want[ok]).max(0) <= 1e-9 * np.abs(want[ok]).max(0))
        far = np.abs(np.tile(hs, len(base)))[ok] >= 1e-2
        assert np.all(np.abs(got - want[ok])[far].max(0) <= 1e-12 * np.abs(want[ok]).max(0))
