"""The ring integrand's shorter form away from the generator and its border to the series form: a charged
circle's field and potential at points with eta = 1 - k^2 on both sides of 0.01, near 1, on the axis and far
away, against scipy's complete elliptic integrals."""

import numpy as np
import pytest
from scipy.special import ellipe, ellipkm1

import kassiopeia_b200 as K
from kassiopeia_b200 import geometry as G

pytestmark = pytest.mark.gpu

R, Z = .7, .2


def points():
    """Points of the plane through the axis at which eta takes given values, at several angles of approach"""
    out = [[0., 0., z] for z in (-3., .2, .2 + 1e-9, 5., 400.)]
    for eta in (1e-6, 5e-3, .01 * (1. - 1e-12), .01, .01 * (1. + 1e-12), .0101, .1, .5, .9, .999999):
        for a in np.linspace(.2, 2. * np.pi, 7):
            # a circle of points with (dr^2 + dz^2) = eta ((R + r)^2 + dz^2), found along the ray of angle a
            lo, hi = 0., 1e4
            for _ in range(200):
                t = .5 * (lo + hi)
                dr, dz = t * np.cos(a), t * np.sin(a)
                r = R + dr
                if r < 0. or t * t > eta * ((R + r) ** 2 + dz * dz):
                    hi = t
                else:
                    lo = t
            out.append([max(0., R + lo * np.cos(a)), 0., Z + lo * np.sin(a)])
    for d in (1e-8, 1e-3, 30., 1e4):
        out += [[d, 0., 0.], [0., d, Z]]
    return np.array(out)


def exact(P):
    r, dz = np.hypot(P[:, 0], P[:, 1]), P[:, 2] - Z
    dr = r - R
    s2 = (R + r) ** 2 + dz ** 2
    eta = (dr ** 2 + dz ** 2) / s2
    m = 4. * R * r / s2
    k, e = ellipkm1(eta), ellipe(m)
    small = m < 1e-4
    # (E - K) / m: its power series where the difference would cancel
    ek = np.where(small, -np.pi / 2 * (.5 + 12. / 64. * m + 30. / 256. * m ** 2 + 1400. / 16384. * m ** 3),
                  (e - k) / np.where(small, 1., m))
    er = (dr * e / eta - 2. * R * ek) / s2 ** 1.5
    ez = dz * e / eta / s2 ** 1.5
    phi = k / np.sqrt(s2)
    u = P[:, :2] / np.maximum(r, 1e-300)[:, None]
    # the terms' sizes; a difference of E and K of relative size m; eta's rounding through dr, amplified by 1 / sqrt(eta)
    size = (np.abs(dr) + np.abs(dz)) * e / eta / s2 ** 1.5 + 2. * R * np.abs(ek) / s2 ** 1.5
    # (to eta = 0.01 the reference's form is kept, which has eta again from a rounded k: eps / eta)
    tol = 1e-14 + 4.4e-16 / np.where(small, 1., m) + 8.8e-16 / np.sqrt(eta) + np.where(eta < .0101, 2.2e-16 / eta, 0.)
    return np.column_stack([er[:, None] * u, ez, phi]), size, tol


def test_ring():
    P = points()
    want, size, tol = exact(P)
    with K.CUDAElectrostaticContext(0) as ctx:
        ctx.SetGeometry(G.axisymmetric(G.RING, np.array([R]), np.array([Z]), value=1.))
        ctx.SetSigma(np.ones(1))
        got = ctx.ElectricFieldAndPotential(P)
        c = got[0, 3] / want[0, 3]  # 1 / (2 pi^2 eps0) times the charge, from the point on the axis
        assert np.all(np.abs(got[:, 3] - c * want[:, 3]) <= tol * np.abs(c * want[:, 3]))
        assert np.all(np.abs(got[:, :3] - c * want[:, :3]) <= (tol * np.abs(c) * size)[:, None])
        for what, sl in ((K.POTENTIAL, slice(3, 4)), (K.FIELD, slice(0, 3))):
            one = ctx.ElectricFieldAndPotential(P, what=what)
            assert np.all(np.abs(one - got)[:, sl] <= (tol * np.abs(c) * np.maximum(size, want[:, 3]))[:, None])
