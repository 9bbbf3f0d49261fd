"""The third-order refinements of the hardware estimates (kemcu_device.cuh: rsqrt_cubic; kemcu_axisym.cuh:
rcp_cubic, sqrt_cubic), restated with exactly rounded fused multiply-adds from estimates off by up to 2^-20,
against the exact values."""

import math
from fractions import Fraction

import numpy as np

from test_cpu_rsqrt import exact_rsqrt, fma


def rsqrt_cubic(x, y):
    e = fma(-(x * y), y, 1.)
    return fma(fma(e, .375, .5), e * y, y)


def rcp_cubic(x, y):
    e = fma(-x, y, 1.)
    return fma(fma(e, e, e), y, y)


def test_third_order_refinements():
    rng = np.random.default_rng(7)
    worst = {"rsqrt": 0., "rcp": 0., "sqrt": 0.}
    for x in np.exp(rng.uniform(np.log(1e-12), np.log(1e12), 500)):
        x = float(x)
        r, root = exact_rsqrt(x), math.sqrt(x)
        for d in (-2. ** -20, 2. ** -20, float(rng.uniform(-2. ** -20, 2. ** -20))):
            a = rsqrt_cubic(x, float(1. / root * (1. + d)))
            b = rcp_cubic(x, float(1. / x * (1. + d)))
            for name, got, want in (("rsqrt", a, r), ("rcp", b, 1 / Fraction(x)), ("sqrt", x * a, r * Fraction(x))):
                worst[name] = max(worst[name], abs(float(Fraction(got) - want)) / math.ulp(float(want)))
    # one rounding of the last step and a fraction of the correction's; the square root adds a product
    assert worst["rsqrt"] <= 1. and worst["rcp"] <= 1. and worst["sqrt"] <= 2., worst
