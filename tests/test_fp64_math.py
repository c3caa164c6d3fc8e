"""The FRU substep's FP64 division and exponential (gw_fp64_math.cuh).

The two-instruction quotient by a constant is correctly rounded for every
operand: the quotients whose distance from a midpoint between two doubles is
within 32 times the form's error are found by modular arithmetic and checked
one by one.  The general quotient and reciprocal are known to 2^-90 before
their last rounding, so one in about 2^36 may differ from the IEEE quotient;
2^30 of each are compared with the hardware's.  The exponential's error is
0.5 ulp of the last rounding, 2^-59.6 of the polynomial (0.011 ulp) and
under 0.005 ulp of the products before it: at most 0.52 ulp."""
import math
import os
import re
from fractions import Fraction as F

import numpy as np
import pytest

from conftest import ROOT

HEADER = os.path.join(ROOT, "greenstein2002_gb300", "csrc", "gw_fp64_math.cuh")
DIVISORS = {"kDiv5": 5.0, "kDiv12": 12.0, "kDivBL": 1.9356, "kDivKrate": 0.00127215, "kDivKrate2": 3.4188,
            "kDivTauss2ss": 10.0 * 0.005, "kDivTauxfer": 0.005, "kDivTautr": 3.0, "kDivRTF": 8.314 * 310.0 / 96.5}


def constants():
    got = re.findall(r"GW_CONST_DIV\((\w+), (-?0x[0-9a-fp.+-]+), (-?0x[0-9a-fp.+-]+)\)", open(HEADER).read())
    return {n: (float.fromhex(h), float.fromhex(l)) for n, h, l in got}


def close_mantissas(d, width):
    """53-bit X whose quotient X/d lies within width/(2D) ulp of a midpoint (D the integer mantissa of d)."""
    D = int(math.frexp(d)[0] * 2 ** 53)
    for s in (52, 53):  # the quotient X 2^s / D has 53 bits: s = 53 where X < D
        A, mod = 1 << (s + 1), 2 * D
        for delta in range(-width, width + 1):
            rhs = (D + delta) % mod
            g = math.gcd(A, mod)
            if delta == 0 or rhs % g:
                continue
            m = mod // g
            x = rhs // g * pow(A // g, -1, m) % m
            x += (2 ** 52 - x + m - 1) // m * m
            while x < 2 ** 53:
                if (x < D) == (s == 53):
                    yield x
                x += m


@pytest.mark.parametrize("name", sorted(DIVISORS))
def test_constant_quotient_is_correctly_rounded(name):
    d = DIVISORS[name]
    hi, lo = constants()[name]
    assert hi == float(1 / F(d)) and lo == float(1 / F(d) - F(hi))
    # the sum x*hi + RN(x*lo) is within err ulp of x/d before the last rounding
    ulp = 2.0 ** (math.floor(math.log2(2 ** 52 / d)) - 52)
    err = 2 ** 53 * (abs(F(lo)) / 2 ** 53 + abs(1 / F(d) - F(hi) - F(lo))) / F(ulp)
    D = int(math.frexp(d)[0] * 2 ** 53)
    assert err * 2 * D < 2  # so width 2 would do
    for x in close_mantissas(d, 64):
        assert float(F(x) * F(hi) + F(float(F(x) * F(lo)))) == float(F(x) / F(d)), x


@pytest.mark.gpu
def test_quotients_match_hardware(gw):
    for seed in (1, 2, 3, 4):
        assert gw.fp64_math_mismatches(1 << 28, seed=seed) == (0, 0, 0)


@pytest.mark.gpu
def test_exp_error(gw):
    rng = np.random.default_rng(11)
    v = np.concatenate([rng.uniform(-140.0, 100.0, 200000), rng.normal(0.0, 1e-4, 20000), [0.0, 35.0, -30.0, -12.5]])
    x = np.concatenate([0.012 * (v - 35.0), -0.05 * (v - 35.0), (v + 12.5) / 5.0, (v + 30.0) / 12.0, 2.0 * v / 26.7,
                        rng.uniform(-599.9, 599.9, 200000)])
    y, _ = gw.exp_device_and_host(x)
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no wider host type")
    true = np.exp(x.astype(np.longdouble))
    err = np.abs((y.astype(np.longdouble) - true) / np.spacing(y))
    print("largest error %.4f ulp" % float(err.max()))
    assert err.max() <= 0.52
    edge = np.array([600.0, -600.0, 709.0, -745.0, 710.0, -746.0, np.inf, -np.inf, np.nan])
    ye, _ = gw.exp_device_and_host(edge)
    np.testing.assert_allclose(ye, np.exp(edge), rtol=1e-15, atol=5e-324)
