"""Point counts around the rounding of the Morton-sort workspace (kemcu_field_dev): every remainder
of its 256-byte regions fits and gives the field of the same points in any other batch."""

import numpy as np
import pytest

import kassiopeia_b200 as K
from kassiopeia_b200 import geometry as G

pytestmark = pytest.mark.gpu


def test_every_remainder_of_the_sort_workspace():
    m = G.icosphere(1)
    P = G.shell_points(4096 + 64, seed=5)
    with K.CUDAElectrostaticContext(0) as ctx:
        ctx.SetGeometry(m)
        ctx.SetSigma(G.sphere_density(m, seed=3))
        want = np.concatenate([ctx.ElectricFieldAndPotential(P[:2000]), ctx.ElectricFieldAndPotential(P[2000:])])
    for r in range(64):
        with K.CUDAElectrostaticContext(0) as ctx:  # a workspace of exactly this count
            ctx.SetGeometry(m)
            ctx.SetSigma(G.sphere_density(m, seed=3))
            out = ctx.ElectricFieldAndPotential(P[:4096 + r])
        # the same pairs in the same element order; the split of the element list may differ
        assert np.max(np.abs(out - want[:4096 + r])) <= 1e-13 * np.max(np.abs(want))
