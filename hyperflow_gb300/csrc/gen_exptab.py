#!/usr/bin/env python3
"""Writes hf_exptab.h: the tables of the short exponential and logarithm of hf_cell.cuh,
the doubles nearest to the exact values (decimal arithmetic at 60 digits)."""
import os
from decimal import Decimal, getcontext

getcontext().prec = 60
HERE = os.path.dirname(os.path.abspath(__file__))
NE, NL = 2048, 256
LN2 = Decimal(2).ln()


def split(v, bits):
    """v = hi + lo with hi a double of at most `bits` significant bits."""
    e = 0
    while abs(v) * (Decimal(2) ** e) < (1 << (bits - 1)):
        e += 1
    hi = Decimal(int((v * Decimal(2) ** e).to_integral_value())) / Decimal(2) ** e
    return float(hi), float(v - hi)


def text():
    exp_tab = [float((Decimal(j) * LN2 / NE).exp()) for j in range(NE)]
    F = [1 + (Decimal(j) + Decimal("0.5")) / NL for j in range(NL)]
    step = LN2 / NE
    # k up to 21 bits: k * STEP_HI is exact; LN2_HI likewise for exponents of 11 bits
    hi, lo = split(step, 32)
    l_hi, l_lo = split(LN2, 42)
    r = step * Decimal("0.51")  # C2 fits this far; the reduced argument reaches 0.65 of a step
    c2 = float(Decimal("0.5") + r * r / 24)
    out = ["// Written by gen_exptab.py: tables of the short exponential and logarithm (hf_cell.cuh).",
           "#pragma once", "namespace hf {", "namespace et {",
           "constexpr double STEP_HI = %s;  // ln2 / %d = HI + LO" % (hi.hex(), NE),
           "constexpr double STEP_LO = %s;" % lo.hex(),
           "constexpr float INV_STEP = %.9ef;  // %d / ln2" % (float(1 / step), NE),
           "constexpr double C2 = %s;  // 1/2 + R^2/24, R = 0.51 ln2 / %d" % (c2.hex(), NE),
           "constexpr double LN2_HI = %s;" % l_hi.hex(),
           "constexpr double LN2_LO = %s;" % l_lo.hex()]
    for name, vals in (("EXP", exp_tab), ("LOG_IF", [float(1 / f) for f in F]), ("LOG_F", [float(f.ln()) for f in F])):
        out.append("static __device__ const double %s[%d] = {" % (name, len(vals)))
        for i in range(0, len(vals), 4):
            out.append("    " + ", ".join(v.hex() for v in vals[i:i + 4]) + ",")
        out.append("};")
    out += ["}  // namespace et", "}  // namespace hf", ""]
    return "\n".join(out)


if __name__ == "__main__":
    with open(os.path.join(HERE, "hf_exptab.h"), "w") as f:
        f.write(text())
