"""The tables of the short exponential and logarithm (csrc/hf_exptab.h), and their formulas
replayed in exact rational arithmetic (one rounding per fused multiply-add) against libm."""
import math
import os
import re
import sys
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hyperflow_gb300", "csrc")
sys.path.insert(0, CSRC)


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


@pytest.fixture(scope="module")
def tab():
    text = open(os.path.join(CSRC, "hf_exptab.h")).read()
    out = {n: float.fromhex(v) for n, v in re.findall(r"constexpr double (\w+) = (\S+);", text)}
    out["INV_STEP"] = float(re.search(r"INV_STEP = (\S+)f;", text).group(1))
    for n in ("EXP", "LOG_IF", "LOG_F"):
        body = re.search(r"double %s\[\d+\] = \{(.*?)\};" % n, text, re.S).group(1)
        out[n] = [float.fromhex(v) for v in re.findall(r"\S+p[-+]\d+", body.replace(",", " "))]
    return out


def test_tables_are_what_the_generator_writes():
    import gen_exptab
    assert open(os.path.join(CSRC, "hf_exptab.h")).read() == gen_exptab.text()


def reduce(x, t):
    k = int(np.rint(np.float32(x) * np.float32(t["INV_STEP"])))
    r = fma(-float(k), t["STEP_LO"], fma(-float(k), t["STEP_HI"], x))
    assert abs(r) <= 0.62 * math.log(2) / 2048
    return k, r


@pytest.mark.parametrize("lo,hi", [(-1.0, 1.0), (-40.0, 40.0), (-339.9, 339.9)])
def test_exponentials(tab, lo, hi):
    """Within 2 ulp: the table and the result round once each (1 ulp), the polynomial's
    terms below 2^-12 of the result add less than half an ulp."""
    for x in np.random.default_rng(1).uniform(lo, hi, 400):
        x = float(x)
        k, r = reduce(x, tab)
        p = fma(r * r, fma(r, 1.0 / 6.0, tab["C2"]), r)
        a = math.ldexp(fma(tab["EXP"][k & 2047], p, tab["EXP"][k & 2047]), k >> 11)
        r2 = r * r
        o = fma(r, r2 * (1.0 / 6.0), r)
        ep = math.ldexp(fma(tab["EXP"][k & 2047], fma(tab["C2"], r2, o), tab["EXP"][k & 2047]), k >> 11)
        em = math.ldexp(fma(tab["EXP"][-k & 2047], fma(tab["C2"], r2, -o), tab["EXP"][-k & 2047]), -k >> 11)
        for got, ref in ((a, math.exp(x)), (ep, math.exp(x)), (em, math.exp(-x))):
            assert abs(got - ref) <= 2 * math.ulp(ref)


@pytest.mark.parametrize("lo,hi", [(0.9, 1.1), (200.0, 6000.0), (1e-300, 1e-290), (1e-8, 1e8), (1e290, 1e300)])
def test_logarithm(tab, lo, hi):
    """Absolute error below 3e-16 + 1 ulp: the FP32 bracket (relative 2^-22) times u^3 <
    7.5e-9 is 2e-16 at most, the sums round to an ulp of the result."""
    rng = np.random.default_rng(2)
    for x in np.exp(rng.uniform(math.log(lo), math.log(hi), 400)):
        x = float(x)
        f, m = math.frexp(x)
        y, m = 2 * f, m - 1
        j = int((y - 1.0) * 256)
        F = 1.0 + (j + 0.5) / 256
        u = (y - F) * tab["LOG_IF"][j]
        q = float(np.float32(1 / 3) + np.float32(u) * (np.float32(-0.25) + np.float32(0.2) * np.float32(u)))
        l = fma(u * u, fma(u, q, -0.5), u)
        got = fma(float(m), tab["LN2_HI"], tab["LOG_F"][j]) + fma(float(m), tab["LN2_LO"], l)
        ref = math.log(x)
        assert abs(got - ref) <= 3e-16 + math.ulp(ref)
