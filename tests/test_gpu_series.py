"""The direct sum, the matrix-free product and the assembled operator at the edges of their new paths:
element counts around the tiles of the far records, point and row counts around a warp, a CTA and the
few-point kernel, near and far points mixed, all element types, Neumann rows, against the C
restatement of the reference."""

import numpy as np
import pytest

import kassiopeia_b200 as K
from kassiopeia_b200 import geometry as G
from oracle import port

pytestmark = pytest.mark.gpu


def mesh(n, seed):
    """n elements of mixed type in runs and singly, sizes over a factor of 30, a third of them Neumann."""
    rng = np.random.default_rng(seed)
    parts = []
    kinds = np.repeat(rng.integers(0, 3, n), rng.integers(1, 24, n))[:n]
    for k in kinds:
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        s = .3 * 30. ** -rng.random()
        p, a, b = rng.uniform(-1, 1, (1, 3)), s * q[:, :1].T, s * rng.uniform(.1, 1.) * q[:, 1:2].T
        bnd = G.NEUMANN if k < 2 and rng.random() < .33 else G.DIRICHLET
        v = 3. if bnd == G.NEUMANN else rng.uniform(-1, 1)
        if k == 0:
            parts.append(G.triangles_from_vertices(p, p + a, p + b + .3 * a, v, bnd))
        elif k == 1:
            parts.append(G.rectangles_from_corners(p, p + a, p + b, v, bnd))
        else:
            parts.append(G.line_segments(p, p + a, 1e-4, v))
    m = parts[0]
    for x in parts[1:]:
        m = m.concat(x)
    return m, 1e-9 * rng.normal(size=n)


def points(n, seed):
    """half of them among the elements, the rest out to 300 sizes away"""
    rng = np.random.default_rng(seed)
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    return np.where(rng.random(n)[:, None] < .5, 1.2 * u * rng.random((n, 1)), u * 1.2 * 50. ** rng.random((n, 1)))


# FP64: rounding of ~20-node sums and of the element sum, a few 1e-15 of the largest term, over results
# that partly cancel; MIXED one Newton step (1e-13 a term, tripled in the field); FP32 1e-7 a node
TOL = {K.FP64: 2e-13, K.MIXED: 5e-12, K.FP32: 3e-6}


@pytest.mark.parametrize("n_elem", [1, 7, 8, 9, 15, 16, 17, 33, 130, 517])
@pytest.mark.parametrize("n_pts", [1, 8, 9, 33, 127, 129, 300])
def test_field_edges(n_elem, n_pts):
    m, sigma = mesh(n_elem, n_elem)
    P = points(n_pts, n_pts)
    o = port.PortProblem(m)
    o.set_sigma(sigma)
    want = o.field(P)
    scale = np.abs(np.concatenate([o.element_field(k, P)[None] * sigma[k] for k in range(m.n)])).sum(0)
    with K.CUDAElectrostaticContext(0) as ctx:
        ctx.SetGeometry(m)
        ctx.SetSigma(sigma)
        for prec, tol in TOL.items():
            for what, sl in ((K.FIELD_AND_POTENTIAL, slice(0, 4)), (K.POTENTIAL, slice(3, 4)), (K.FIELD, slice(0, 3))):
                out = ctx.ElectricFieldAndPotential(P, precision=prec, what=what)
                # per point, relative to the sum of the terms' sizes (of the field's vector)
                s = np.concatenate([np.repeat(np.linalg.norm(scale[:, :3], axis=1)[:, None], 3, 1), scale[:, 3:]], 1)
                assert np.all(np.abs(out - want)[:, sl] <= tol * s[:, sl]), (prec, what)


@pytest.mark.parametrize("n_elem", [1, 8, 17, 31, 33, 129, 260, 517])
def test_operator_edges(n_elem):
    m, _ = mesh(n_elem, 1000 + n_elem)
    A, _ = port.PortProblem(m).matrix()
    rng = np.random.default_rng(3)
    finite = np.isfinite(A).all(1) & (np.arange(m.n) >= 0)
    # a wire's potential on its own axis has logarithms of R - s with R^2 - s^2 = (diameter / 2)^2: eps
    # (length / diameter)^2 of rounding in each of two, in this code and in the restatement alike
    wire = m.shape == G.LINE_SEGMENT
    own = np.where(wire, 2 * 2.2e-16 * (.3 / 1e-4) ** 2, 0.) * np.abs(np.diag(A))
    with K.CUDAElectrostaticContext(0) as ctx:
        ctx.SetGeometry(m)
        for nr in (1, 2, 8):
            x = rng.normal(size=(nr, m.n))
            want, size, extra = x @ A.T, np.abs(x) @ np.abs(A).T, np.abs(x) * own
            for prec, tol in TOL.items():
                y = ctx.Multiply(x if nr > 1 else x[0], precision=prec).reshape(nr, -1)
                assert np.all(np.abs(y - want)[:, finite] <= (tol * size + extra)[:, finite]), (nr, prec)
            y = ctx.Multiply(x if nr > 1 else x[0], assembled=True).reshape(nr, -1)
            assert np.all(np.abs(y - want)[:, finite] <= (TOL[K.FP64] * size + extra)[:, finite]), nr


def test_degenerate_elements_keep_the_cubature():
    # a triangle without area has no plane for the series; its far field is zero, as before
    m = G.triangles_from_vertices([[0., 0, 0], [1., 0, 0]], [[1., 0, 0], [2., 0, 0]], [[2., 0, 0], [1., 1, 0]], 1.)
    with K.CUDAElectrostaticContext(0) as ctx:
        ctx.SetGeometry(m)
        ctx.SetSigma(np.array([1e-9, 1e-9]))
        P = points(200, 4) * 40. + 60.
        o = port.PortProblem(m)
        o.set_sigma(np.array([1e-9, 1e-9]))
        want = o.field(P)
        assert np.allclose(ctx.ElectricFieldAndPotential(P), want, rtol=1e-12, atol=0)
