"""The argument reduction and the polynomials of the short exponential and logarithm
(csrc/hf_cell.cuh) as the device evaluates them: conversions to FP32 cut toward zero, FP32
products rounded, one rounding per fused multiply-add."""
import math

import numpy as np
import pytest

from test_cell_tables import fma, tab  # noqa: F401

L = np.longdouble
F = np.float32


def to_f32(x):
    """x cut to 24 bits."""
    m, e = math.frexp(x)
    return F(math.ldexp(math.trunc(m * 2 ** 24), e - 24)) if abs(x) >= 2.0 ** -126 else F(math.copysign(0.0, x))


def fmaf(a, b, c):
    return F(float(a) * float(b) + float(c))  # exact in 64 bits but for the last rounding


def reduce(x, t):
    k = int(np.rint(to_f32(x) * F(t["INV_STEP"])))
    return k, fma(-float(k), t["STEP_LO"], fma(-float(k), t["STEP_HI"], x))


def arguments():
    """Random ones, and those next to a half step, where the reduced argument is largest."""
    rng = np.random.default_rng(8)
    mid = (rng.integers(-1000000, 1000000, 3000) + 0.5) * (math.log(2) / 2048)
    x = np.concatenate([mid, mid * (1 + 1e-7), mid * (1 - 1e-7), rng.uniform(-339.9, 339.9, 500), rng.uniform(-30, 30, 500)])
    return [float(v) for v in x if abs(v) < 340]


def test_reduced_argument(tab):  # noqa: F811
    """The cut takes 2^-23 of x, the product rounds to 2^-24 of the quotient: at |x| = 340
    0.12 + 0.03 of a step beyond the half, less where k is small."""
    worst = max(abs(reduce(x, tab)[1]) for x in arguments()) / (math.log(2) / 2048)
    assert 0.55 < worst <= 0.65


def test_exponentials(tab):  # noqa: F811
    for x in arguments()[::4]:
        k, r = reduce(x, tab)
        t, s = tab["EXP"][k & 2047], tab["EXP"][-k & 2047]
        a = math.ldexp(fma(t, fma(r * r, fma(r, 1.0 / 6.0, tab["C2"]), r), t), k >> 11)
        r2 = r * r
        o = fma(r, r2 * (1.0 / 6.0), r)
        ep = math.ldexp(fma(t, fma(tab["C2"], r2, o), t), k >> 11)
        em = math.ldexp(fma(s, fma(tab["C2"], r2, -o), s), -k >> 11)
        for got, ref in ((a, np.exp(L(x))), (ep, np.exp(L(x))), (em, np.exp(-L(x)))):
            assert abs(L(got) - ref) <= L(1.35) * math.ulp(float(ref))


@pytest.mark.parametrize("lo,hi", [(0.5, 2.0), (0.998, 1.002), (200.0, 6000.0), (1e-290, 1e-280)])
def test_logarithm(tab, lo, hi):  # noqa: F811
    for x in np.exp(np.random.default_rng(9).uniform(math.log(lo), math.log(hi), 1500)):
        x = float(x)
        f, m = math.frexp(x)
        y, m = 2 * f, m - 1
        j = int((y - 1.0) * 256)
        u = (y - (1.0 + (j + 0.5) / 256)) * tab["LOG_IF"][j]
        f = to_f32(u)
        q = float(fmaf(f, fmaf(f, F(0.2), F(-0.25)), F(1 / 3)))
        l = fma(u * u, fma(u, q, -0.5), u)
        got = fma(float(m), tab["LN2_HI"], tab["LOG_F"][j]) + fma(float(m), tab["LN2_LO"], l)
        ref = np.log(L(x))
        assert abs(L(got) - ref) <= L(1.5) * math.ulp(float(ref)) + L(2.7e-16)
