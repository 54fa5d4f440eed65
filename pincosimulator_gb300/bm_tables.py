"""Tables of the FP64 Box-Muller draw (csrc/twmc_common.cuh), emitted as
csrc/bm_tables.inc: table-driven logarithm and sine / cosine in the manner of
Tang (ACM Trans. Math. Softw. 16, 1990 and 17, 1991), the logarithm's reduction
that of log in Arm Optimized Routines (math/log.c, MIT licence: offset 0.6875, 128
intervals of the bit pattern, one of them ending at 1), every entry computed
here and rounded once from 60 digits.

The uniforms are u = (w + 1/2) 2^-32, w a 32-bit word.

* -2 ln u: 2 w + 1 = z 2^k with z in [0.6875, 1.375), cut into 128 intervals of
  the bit pattern (tmp = bits - bits(0.6875)); per interval -2 / c (c its
  centre, 1 for the one that ends at 1, so that ln u near 0 keeps its relative
  accuracy) and 2 ln(1 / c) of that rounded reciprocal; per exponent -2 k ln 2.
* cos, sin of 2 pi u - pi: the centres of 256 sectors.
"""
from __future__ import annotations

import struct
from decimal import Decimal, getcontext

getcontext().prec = 60

PI = Decimal("3.14159265358979323846264338327950288419716939937510582097494459")
LN2 = Decimal(2).ln()


def _bits(x: float) -> int:
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def _float(b: int) -> float:
    return struct.unpack("<d", struct.pack("<Q", b))[0]


def cossin(x: Decimal):
    """(cos, sin) of |x| <= pi by Taylor series."""
    c = s = Decimal(0)
    term, n = Decimal(1), 0
    while abs(term) > Decimal(10) ** -58:
        if n % 2 == 0:
            c += term if n % 4 == 0 else -term
        else:
            s += term if n % 4 == 1 else -term
        n += 1
        term = term * x / n
    return c, s


OFF = 0.6875


def log_table():
    """[(-2 / c, 2 ln c)] for the 128 intervals (signs folded: the sum with the
    polynomial in s = 2 - 2 z / c is -2 ln z)."""
    out = []
    base, step = _bits(OFF), 1 << (52 - 7)
    for i in range(128):
        lo, hi = _float(base + i * step), _float(base + (i + 1) * step)
        c = Decimal(1) if hi == 1.0 else (Decimal(lo) + Decimal(hi)) / 2
        inv = float(1 / c)
        out.append((-2.0 * inv, float(2 * Decimal(inv).ln()) if inv != 1.0 else 0.0))
    return out


def exponent_table():
    """-2 k ln 2 for k = -33 .. 0."""
    return [float(-2 * k * LN2) for k in range(-33, 1)]


def sector_table():
    """(cos, sin) at 2 pi ((i + 1/2) / 256 - 1/2)."""
    out = []
    for i in range(256):
        c, s = cossin(2 * PI * ((Decimal(i) + Decimal("0.5")) / 256 - Decimal("0.5")))
        out.append((float(c), float(s)))
    return out


def emit_header() -> str:
    def pairs(name, t):
        body = ",\n    ".join("{%s, %s}" % (a.hex(), b.hex()) for a, b in t)
        return f"static __device__ const double2 {name}[{len(t)}] = {{\n    {body}}};\n"

    exps = ",\n    ".join(v.hex() for v in exponent_table())
    return ("// Generated by pincosimulator_gb300/bm_tables.py -- do not edit.\n#pragma once\nnamespace twmc {\n" +
            pairs("kLogTable", log_table()) + pairs("kSectorTable", sector_table()) +
            f"static __device__ const double kExpTable[34] = {{\n    {exps}}};\n" + "}  // namespace twmc\n")
