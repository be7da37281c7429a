"""Writes the constants of vh_crmath.cuh: ln 2 split into three doubles (the
first with 33 significant bits, so that k * LN2_1 is exact for |k| < 2^20),
1 / ln 2 rounded to nearest, and 1/n! (n = 2..11) as double-double pairs.
Exact rational arithmetic (fractions) and a 60-digit decimal ln 2
(decimal.Decimal.ln); run it to check the literals in the header:

    python vhlle_b200/csrc/gen_crmath_consts.py

It also writes vh_crmath_tab.cuh: for exp's and log's short forms ln 2 and
ln 2 / 64 in two doubles, 2^(j/64) and, per 1/128 of [1, 2), the reciprocal
of the middle and minus its logarithm as double-double pairs.
"""
import decimal
import math
import os
from fractions import Fraction

decimal.getcontext().prec = 80
LN2 = Fraction(decimal.Decimal(2).ln())


def rn(q: Fraction) -> float:
    """q rounded to the nearest double (ties to even), via float(Fraction)."""
    return float(q)


def trunc_bits(q: Fraction, bits: int) -> float:
    """q > 0 truncated to `bits` significant bits (a double)."""
    exp = math.frexp(float(q))[1]
    scale = Fraction(2) ** (bits - exp)
    return float(Fraction(int(q * scale)) / scale)


def main():
    l1 = trunc_bits(LN2, 33)
    r = LN2 - Fraction(l1)
    l2 = rn(r)
    r -= Fraction(l2)
    l3 = rn(r)
    print("LN2_1 = %s  // %r" % (l1.hex(), l1))
    print("LN2_2 = %s  // %r" % (l2.hex(), l2))
    print("LN2_3 = %s  // %r" % (l3.hex(), l3))
    print("INV_LN2 = %s" % rn(1 / LN2).hex())
    f = Fraction(1)
    for n in range(1, 12):
        f /= n
        hi = rn(f)
        lo = rn(f - Fraction(hi))
        print("INV_FACT[%d] = {%s, %s}" % (n, hi.hex(), lo.hex()))


def pair(q: Fraction):
    hi = rn(q)
    return hi, rn(q - Fraction(hi))


def tables():
    dec = lambda q: decimal.Decimal(q.numerator) / decimal.Decimal(q.denominator)  # noqa: E731
    out = ["// Written by gen_crmath_consts.py: the tables of vh_crmath.cuh's short forms.",
           "#pragma once", ""]
    for name, q, bits in (("LN2", LN2, 42), ("LN2_64", LN2 / 64, 36)):
        h = trunc_bits(q, bits)
        out.append("#define VH_CRM_%sH %s" % (name, h.hex()))
        out.append("#define VH_CRM_%sL %s" % (name, rn(q - Fraction(h)).hex()))
    out.append("#define VH_CRM_64_LN2 %s" % rn(64 / LN2).hex())
    exp2 = [pair(Fraction((decimal.Decimal(j) / 64 * decimal.Decimal(2).ln()).exp())) for j in range(64)]
    logs = []
    for i in range(128):
        c = rn(1 / (1 + Fraction(2 * i + 1, 256)))
        logs.append((c,) + pair(-Fraction(dec(Fraction(c)).ln())))
    for name, rows in (("EXP_TAB", exp2), ("LOG_TAB", logs)):
        out.append("#define VH_CRM_%s \\" % name)
        out += ["  " + ", ".join(float(v).hex() for v in r) + (", \\" if r is not rows[-1] else "") for r in rows]
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), "vh_crmath_tab.cuh")
    with open(path, "w") as f:
        f.write("\n".join(out) + "\n")


if __name__ == "__main__":
    main()
    tables()
