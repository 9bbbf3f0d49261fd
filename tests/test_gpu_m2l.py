"""M2L on the tensor cores: one, two, seven and eight right-hand sides (different column layouts of the
same product) agree, at degrees around the 8-row fragments and the two-tile warps, on trees with
different divisions, top levels and neighbour orders, and with the products of a tree whose offset lists
are too long for it (the kernel that walks the neighbourhood)."""

import numpy as np
import pytest

import kassiopeia_b200 as K
from kassiopeia_b200 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree,depth,divisions,top,zeromask", [
    (0, 3, 2, 2, 1), (1, 3, 2, 1, 1), (2, 4, 2, 2, 1), (7, 3, 2, 2, 1), (8, 3, 2, 3, 1), (8, 3, 3, 2, 1), (6, 3, 2, 2, 2),
    (11, 3, 2, 2, 1), (15, 2, 2, 2, 1), (4, 2, 4, 2, 1)])
def test_columns_agree(degree, depth, divisions, top, zeromask):
    m = G.stacked_rings(n_rings=4, n_phi=24, n_z=8)
    rng = np.random.default_rng(degree)
    x = rng.normal(size=(8, m.n))
    with K.CUDAElectrostaticContext(0) as ctx:
        ctx.SetGeometry(m)
        ctx.ConfigureFFTM(degree=degree, maximum_tree_depth=depth, divisions=divisions, top_level_divisions=top,
                          zeromask=zeromask)
        one = np.stack([ctx.FFTMMultiply(x[r]) for r in range(8)])
        # sums of the same products in another order: rounding of a few hundred terms
        for nr in (2, 7, 8):
            y = ctx.FFTMMultiply(x[:nr])
            assert np.max(np.abs(y - one[:nr])) <= 1e-13 * np.max(np.abs(one))
        direct = ctx.Multiply(x[0])
        # the truncated expansions' error falls with the degree (loose: a wrong interaction is 1e-1)
        assert np.linalg.norm(one[0] - direct) <= (.5 if degree == 0 else .1 if degree < 4 else 5e-3) * np.linalg.norm(direct)


def test_neighbourhood_walk_gives_the_same_operator():
    # divisions 8 below a single top cell (offset lists of seven million entries) and top_level_divisions 8
    # with one level: the same leaves, neighbours and interactions
    m = G.icosphere(2)
    x = np.random.default_rng(2).normal(size=(3, m.n))
    out = []
    for kw in (dict(maximum_tree_depth=2, top_level_divisions=1, divisions=8), dict(maximum_tree_depth=1, top_level_divisions=8)):
        with K.CUDAElectrostaticContext(0) as ctx:
            ctx.SetGeometry(m)
            ctx.ConfigureFFTM(degree=3, **kw)
            out.append(np.concatenate([ctx.FFTMMultiply(x), [ctx.FFTMMultiply(x[0])]]))
    assert np.max(np.abs(out[0] - out[1])) <= 1e-13 * np.max(np.abs(out[0]))


@pytest.mark.parametrize("n", [1, 31, 700])
def test_field_uses_the_same_expansions(n):
    # the field's tiles are built on the device from the points' leaves; the product's on the host
    m = G.icosphere(3)
    s = G.sphere_density(m, seed=4)
    P = G.shell_points(n, r_min=1.0, seed=n) * .98
    with K.CUDAElectrostaticContext(0) as ctx:
        ctx.SetGeometry(m)
        ctx.SetSigma(s)
        ctx.ConfigureFFTM(degree=8, maximum_tree_depth=3)
        out = ctx.FFTMField(P)
        want = ctx.ElectricFieldAndPotential(P)
        assert np.max(np.abs(out - want)) <= 5e-3 * np.max(np.abs(want))
