"""Single pairs of the three precision forms over every distance from the analytic band to beyond the last cut of
the far-field series, each point in a warp of its own, so that its own distance decides: a sum over many
elements hides what one pair loses."""

import numpy as np
import pytest

import kassiopeia_b200 as K
from kassiopeia_b200 import geometry as G

pytestmark = pytest.mark.gpu


def pairs(shape, a, b, n=3000):
    """fields of one element at n points, in FP64, MIXED and FP32, as (error against FP64, per point) of the latter two"""
    rng = np.random.default_rng(int(shape) + 7)
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    a, b, p0 = q[:, :2] @ np.array(a), q[:, :2] @ np.array(b), np.zeros((1, 3))
    if shape == G.TRIANGLE:
        m, size = G.triangles_from_vertices(p0, p0 + a, p0 + b, 1.), (np.linalg.norm(a) + np.linalg.norm(b) + np.linalg.norm(a - b)) / 3
    elif shape == G.RECTANGLE:
        m, size = G.rectangles_from_corners(p0, p0 + a, p0 + b, 1.), .5 * (np.linalg.norm(a) + np.linalg.norm(b))
    else:
        m, size = G.line_segments(p0, p0 + a, 1e-4, 1.), np.linalg.norm(a)
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    P = .5 * (a + b) + u * (size * np.exp(rng.uniform(np.log(5.), np.log(300.), n)))[:, None]
    out = {}
    with K.CUDAElectrostaticContext(0) as ctx:
        ctx.SetGeometry(m)
        ctx.SetSigma(np.ones(1))
        for form in (K.FP64, K.MIXED, K.FP32):
            out[form] = ctx.ElectricFieldAndPotential(np.repeat(P, 32, axis=0), precision=form)[::32]
    want = out[K.FP64]
    return {f: np.stack([np.linalg.norm(out[f][:, :3] - want[:, :3], axis=1) / np.linalg.norm(want[:, :3], axis=1),
                         np.abs(out[f][:, 3] / want[:, 3] - 1)]) for f in (K.MIXED, K.FP32)}


@pytest.mark.parametrize("a", [[1., 0.], [1e-3, 0.]])
def test_wires_are_fp64_in_every_form(a):
    for e in pairs(G.LINE_SEGMENT, a, [0., 0.]).values():
        # rounding of both forms, the first orders left out and the FP32 tail, a few 1e-15 in the worst direction
        assert e.max() <= 1e-14, e.max(1)


@pytest.mark.parametrize("shape,a,b", [(G.TRIANGLE, [1., 0.], [.5, .866]), (G.TRIANGLE, [1., 0.], [.02, .07]),
                                       (G.RECTANGLE, [1., 0.], [0., 1.]), (G.RECTANGLE, [1., 0.], [.6, .8])])
def test_mixed_pairs(shape, a, b):
    e = pairs(shape, a, b)
    # a node's reciprocal distance is within 1.3e-12 (one Newton step from the hardware's estimate), its cube, the
    # field's, within 3.9e-12; a rule averages 7 to 33 of them with errors of both signs, and the series has 3e-13
    # of its FP32 orders: never above half of a node's bound, and a quarter of a node's typical error in the mean
    assert e[K.MIXED][0].max() <= 2e-12 and e[K.MIXED][1].max() <= 6.5e-13, e[K.MIXED].max(1)
    assert np.sqrt((e[K.MIXED][0] ** 2).mean()) <= 4e-13 and np.sqrt((e[K.MIXED][1] ** 2).mean()) <= 1.1e-13
    assert e[K.FP32].max() <= 1e-6
