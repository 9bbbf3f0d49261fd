"""Robin Hood on one CTA at the edges of its row layout (a warp, a CTA, two and four rows a thread, and
past it), columns assembled and asked to be computed on the fly: the direct solution, and the same
solution and corrections however the columns come."""

import numpy as np
import pytest

import kassiopeia_b200 as K
from kassiopeia_b200 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 320, 1023, 1025, 1280, 2049, 4096, 4100])
def test_row_layouts(n):
    full = G.icosphere(4)
    m = G.Mesh(full.shape[:n], full.boundary[:n], full.geom[:n], full.value[:n])
    rng = np.random.default_rng(n)
    b = 1. + .3 * rng.normal(size=n)
    with K.CUDAElectrostaticContext(0) as ctx:
        ctx.SetGeometry(m)
        x, st = ctx.SolveRobinHood(b, tol=1e-7)
        y, st2 = ctx.SolveRobinHood(b, tol=1e-7, assembled=True)
        # |b - A x|_inf / |b|_inf at a check is at most the tolerance; one more correction may follow
        for v in (x, y):
            assert np.max(np.abs(b - ctx.Multiply(v))) <= 2e-7 * np.max(np.abs(b))
        assert st["iterations"] == st2["iterations"]
        # the starting guess is kept: from the solution itself the first check ends the solve
        z, st3 = ctx.SolveRobinHood(b, tol=1e-6, x0=x)
        assert st3["iterations"] == 1 and np.max(np.abs(z - x)) <= 1e-5 * np.max(np.abs(x))


def test_budget_too_small_for_the_operator_keeps_columns_on_the_fly():
    m = G.icosphere(2)
    b = np.ones(m.n)
    with K.CUDAElectrostaticContext(0, assembled_budget_bytes=1000) as ctx:
        ctx.SetGeometry(m)
        x, _ = ctx.SolveRobinHood(b, tol=1e-7)
        assert np.max(np.abs(b - ctx.Multiply(x))) <= 2e-7
