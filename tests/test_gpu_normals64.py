"""The FP64 Box-Muller draw on the device against 60 digits.

Bound of one draw, in units of u = 2^-53 and of its radius r = sqrt(-2 ln u1):
-2 ln u1 is good to 3 u (tests/test_bm_tables.py), its root to half of that and a
rounding of u, cos and sin to 2 u absolutely (the same test), the product to
another u: 1.5 + 1 + 2 + 1 = 5.5. Over a sample the errors are no larger than
those of the library's log, sqrt and sincos that the tables took the place
of: rms 1.41e-16, at most 1.09e-15 over 8192 pairs."""
from decimal import Decimal

import numpy as np
import pytest

from pincosimulator_gb300 import bm_tables as bm
from pincosimulator_gb300 import twmc

pytestmark = pytest.mark.gpu

WIENER_KEY = (0x243F6A88, 0x85A308D3)


def test_draws_against_60_digits(built_lib):
    n, steps, seed, tid = 2048, 4, 77, 5
    half = n // 2
    xi = twmc.debug_wiener(twmc.PREC_F64, seed, tid, steps, n, step0=100)
    sq, worst, most = 0.0, 0.0, 0.0
    for k in range(steps):
        ctr = np.array([(p, 100 + k, tid, seed) for p in range(half)], dtype=np.uint32)
        words = twmc.debug_philox(ctr, WIENER_KEY)
        for site in range(n):
            a, b = (int(w) for w in words[site % half][2 * (site // half):2 * (site // half) + 2])
            r = (-2 * (Decimal(2 * a + 1) / 2 ** 33).ln()).sqrt()
            c, s = bm.cossin(2 * bm.PI * (Decimal(2 * b + 1) / 2 ** 33) - bm.PI)
            got = xi[k, site]
            for v, ref in ((got.real, r * c), (got.imag, r * s)):
                e = float(abs(Decimal(float(v)) - ref))
                worst = max(worst, e / float(r))
                most = max(most, e)
                sq += e * e
    rms = (sq / (2 * n * steps)) ** 0.5
    print(f"rms {rms:.3e}, largest {most:.3e}, largest / r {worst * 2 ** 53:.2f} u")
    assert worst <= 5.5 * 2.0 ** -53
    assert rms <= 1.41e-16 and most <= 1.09e-15
