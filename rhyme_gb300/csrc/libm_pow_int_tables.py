"""Writes libm_pow_int_tables.h: the constants of libm_pow_int.h.

    python rhyme_gb300/csrc/libm_pow_int_tables.py [OUT]

Every value is one of libm_pow_tables.h's doubles (or a sum of two of them),
scaled by a power of two and rounded to the nearest integer:
  LOG[i]   LOGC + LOGCTAIL of piece i in units of 2^-78 (low 64 bits, high 64
           bits), and 256 INVC, an integer below 363;
  LN2      LN2_HI + LN2_LO in units of 2^-78;
  B1..B6   the coefficients of (log1p(r) - r + r^2/2)/r^3 as one polynomial in
           r: with libm_pow.h's A1..A6, -A1/2, -A2/2, A3/4, A4/4, -A5/8,
           -A6/8; B1..B3 in units of 2^-63, B4..B6 of 2^-33;
  HL       -(NEG_LN2_HI_N + NEG_LN2_LO_N), ln 2 / 128, in units of 2^-92;
  LO       -NEG_LN2_LO_N in units of 2^-95;
  INV      INV_LN2_N in units of 2^-20.
"""
import os
import re
import sys
from fractions import Fraction

HERE = os.path.dirname(os.path.abspath(__file__))


def main(out=None):
    text = open(os.path.join(HERE, "libm_pow_tables.h")).read()
    value = lambda s: Fraction(float.fromhex(s))  # noqa: E731
    number = r"(-?(?:0x\S+|0\.0))"
    log = text[text.index("LIBM_POW_LOG_TABLE {"):text.index("LIBM_POW_EXP_TABLE {")]
    rows = re.findall(r"^ +%s, %s, %s, 0\.0," % (number, number, number), log, re.M)
    assert len(rows) == 128
    c = {n: value(v) for n, v in re.findall(r"constexpr double LIBM_POW_(\w+) = (\S+);", text)}

    def units(v, bits):
        return (v * 2 ** bits + Fraction(1, 2)).__floor__()

    def halves(v):
        return "0x%016xULL, %dLL" % (v & (2 ** 64 - 1), v >> 64)

    lines = ["// libm_pow_int_tables.h -- constants of libm_pow_int.h, written by",
             "// libm_pow_int_tables.py; do not edit by hand.", "#pragma once", "",
             "#define LIBM_POW_INT_LOG { \\"]
    for invc, logc, tail in rows:
        assert (value(invc) * 256).denominator == 1
        lines.append("    {%s, %d}, \\" % (halves(units(value(logc) + value(tail), 78)), int(value(invc) * 256)))
    lines.append("}")
    lines.append("#define LIBM_POW_INT_LN2 %s" % halves(units(c["LN2_HI"] + c["LN2_LO"], 78)))
    b = [-c["A1"] / 2, -c["A2"] / 2, c["A3"] / 4, c["A4"] / 4, -c["A5"] / 8, -c["A6"] / 8]
    for i, v in enumerate(b):
        lines.append("constexpr int64_t LIBM_POW_INT_B%d = %dLL;" % (i + 1, units(v, 63 if i < 3 else 33)))
    lines.append("#define LIBM_POW_INT_HL %s" % halves(units(-(c["NEG_LN2_HI_N"] + c["NEG_LN2_LO_N"]), 92)))
    lines.append("constexpr int64_t LIBM_POW_INT_LO = %dLL;" % units(-c["NEG_LN2_LO_N"], 95))
    lines.append("constexpr int64_t LIBM_POW_INT_INV = %dLL;" % units(c["INV_LN2_N"], 20))
    out = out or os.path.join(HERE, "libm_pow_int_tables.h")
    with open(out, "w") as f:
        f.write("\n".join(lines) + "\n")
    print("wrote", out)


if __name__ == "__main__":
    main(sys.argv[1] if len(sys.argv) > 1 else None)
