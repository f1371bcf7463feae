"""Writes qj_fxmath_tables.h: the tables of the fixed-point transcendentals in
qj_fxmath.h, computed here with mpmath at 300 bits and rounded to nearest.

    python quijibo_gb300/csrc/gen_fxmath_tables.py

Every value is a power of two, logarithm, sine, cosine or arcsine at a table
point, so the file is the same on every machine that runs this script.
"""
import os

import mpmath

mpmath.mp.prec = 300


def fix(v, bits):
    """v as an integer of 2^-bits units."""
    return int(mpmath.nint(mpmath.ldexp(v, bits)))


def main():
    out = []
    w = out.append
    w("// Generated by gen_fxmath_tables.py (mpmath, 300 bits): do not edit.")
    w("#pragma once")
    w("")

    def table(name, doc, rows):
        w("// %s" % doc)
        w("FX_TAB fx_pair %s[%d] = {" % (name, len(rows)))
        for a, b in rows:
            w("    {0x%016xull, 0x%016xull}," % (a & (1 << 64) - 1, b & (1 << 64) - 1))
        w("};")
        w("")

    rows = []
    for j in range(256):
        mid = 1 + mpmath.mpf(2 * j + 1) / 512
        c = int(mpmath.nint(mpmath.mpf(2048) / mid))  # 1/m in 2^-11
        k = 1 if j >= 106 else 0  # m > sqrt(2): log(m / 2), the exponent raised by one
        rows.append((fix(-mpmath.log(mpmath.mpf(c) / 2048) - k * mpmath.log(2), 63), c | k << 16))
    table("fx_tab_log", "{-log(c) - k log 2 in 2^-63, c in 2^-11 | k << 16}, c about 1/m", rows)
    rows = [(fix(mpmath.mpf(2) ** (mpmath.mpf(j) / 256), 63), 0) for j in range(256)]
    w("// 2^(j/256) in 2^-63")
    w("FX_TAB unsigned long long fx_tab_exp[256] = {")
    for a, _ in rows:
        w("    0x%016xull," % a)
    w("};")
    w("")
    rows = []
    for j in range(257):
        t = mpmath.pi * j / 512
        rows.append((fix(mpmath.sin(t), 62), fix(mpmath.cos(t), 62)))
    table("fx_tab_sin", "{sin, cos} of j pi/512 in 2^-62", rows)
    rows = []
    for j in range(363):
        a = mpmath.mpf(2 * j + 1) / 1024
        rows.append((fix(mpmath.asin(a), 62), fix(mpmath.sqrt(1 - a * a), 64)))
    table("fx_tab_asin", "{asin(a) in 2^-62, sqrt(1 - a^2) in 2^-64}, a = (2j + 1)/1024", rows)
    with open(os.path.join(os.path.dirname(os.path.abspath(__file__)), "qj_fxmath_tables.h"), "w") as f:
        f.write("\n".join(out))


if __name__ == "__main__":
    main()
