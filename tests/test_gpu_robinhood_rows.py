"""Robin Hood on one CTA at the edges of its row layout (a warp, a CTA, two and four rows a thread, and
past it), columns assembled and asked to be computed on the fly: the direct solution, and the same
solution and corrections however the columns come."""

import numpy as np
import pytest

import kassiopeia_b200 as K
from kassiopeia_b200 import geometry as G
from oracle import golden

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


@pytest.mark.parametrize("name", ["icosphere_L2", "mixed_small", "c1_sphere"])
def test_columns_on_the_fly_match_the_reference(name):
    # no room for kept columns: one CTA, or (1,280 rows) a cluster, computes every column (near list and cubature
    # bands; mixed_small has Neumann rows and wires); the reference's number of checks, and its solution
    tol = 1e-8
    fx = golden.load(name)
    if name == "c1_sphere":
        m, checks, sigma, direct = G.icosphere(3), fx["robinhood_iterations"], fx["robinhood_sigma"], fx["sigma_direct"]
    else:
        rh = golden.load("robinhood")
        m, checks, sigma = golden.mesh_from(fx), rh[f"{name}_{tol:.0e}_iterations"], rh[f"{name}_{tol:.0e}_sigma"]
        direct = fx["sigma_direct" if name == "icosphere_L2" else "x_direct"]

    def rel(a, b):
        return np.max(np.abs(a - b)) / np.max(np.abs(b))
    bound = max(5 * rel(sigma, direct), 100 * tol)
    with K.CUDAElectrostaticContext(0, assembled_budget_bytes=8) as ctx:
        ctx.SetGeometry(m)
        x, st = ctx.SolveRobinHood(tol=tol)
        assert st["rel_residual"] <= tol and abs(st["iterations"] - int(checks)) <= 1
        assert rel(x, direct) <= bound and rel(x, sigma) <= bound
        with pytest.raises(K.KemcuError):  # the budget is the caller's
            ctx.SolveRobinHood(tol=tol, assembled=True)
    with K.CUDAElectrostaticContext(0) as ctx:  # kept columns: entries of another quadrature, 1e-14 apart
        ctx.SetGeometry(m)
        y, st2 = ctx.SolveRobinHood(tol=tol)
        assert abs(st2["iterations"] - st["iterations"]) <= 1 and rel(y, x) <= 2 * bound


def test_kept_columns_end_with_the_solve():
    torch = pytest.importorskip("torch")
    full = G.icosphere(4)
    n = 3000  # 72 MB of columns
    m = G.Mesh(full.shape[:n], full.boundary[:n], full.geom[:n], full.value[:n])
    with K.CUDAElectrostaticContext(0) as ctx:
        ctx.SetGeometry(m)
        ctx.SolveRobinHood(np.ones(n), tol=1e-3, max_subiterations=10, raise_on_failure=False, assembled=False)
        free = torch.cuda.mem_get_info()[0]
        ctx.SetGeometry(m)
        ctx.Multiply(np.ones(n), assembled=True)
        held = free - torch.cuda.mem_get_info()[0]
        assert held > 60e6  # the operator that was asked for; the solve had kept none
        ctx.SolveRobinHood(np.ones(n), tol=1e-3, max_subiterations=10, raise_on_failure=False)
        assert free - torch.cuda.mem_get_info()[0] > 60e6  # and leaves it
