"""A track's bits do not depend on the tracks beside it: alone, in a batch for every number of warps that the
tracker gives a CTA (16, 8 and 4 from the number of tracks), and in another order of the list."""

import numpy as np
import pytest

import kassiopeia_b200 as K
from kassiopeia_b200 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [K.FP64, K.MIXED])
@pytest.mark.parametrize("n_elem", [1, 15, 17, 80])  # fewer parts than warps, and around them
def test_batches_give_the_same_bits(precision, n_elem):
    full = G.icosphere(1)
    m = G.Mesh(full.shape[:n_elem], full.boundary[:n_elem], full.geom[:n_elem], full.value[:n_elem])
    state = G.electrons(16384, seed=5)
    with K.CUDAElectrostaticContext(0) as ctx:
        ctx.SetGeometry(m)
        ctx.SetSigma(1e-9 * np.random.default_rng(1).normal(size=m.n))

        def run(st):
            return ctx.TrackRK8(st, 1e-11, 100, step_budget=2, precision=precision)[0]
        want = run(state)
        assert np.any(want[:, 5:] != state[:, 5:])
        for n in (1, 2, 33, 600, 6000):
            assert np.array_equal(run(state[:n]), want[:n]), n
        assert np.array_equal(run(state[::-1]), want[::-1])
