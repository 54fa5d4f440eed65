"""Tables of the FP64 Box-Muller draw: the device's arithmetic restated with
exact products (one rounding per multiply-add) against 60 digits, on random
words and on those at the edges of the reductions."""
import random
from decimal import Decimal

from pincosimulator_gb300 import bm_tables as bm

U = Decimal(2) ** -53
EDGES = [0, 1, 2, 3, 2**31 - 1, 2**31, 2**32 - 2, 2**32 - 1, 0x00ffffff, 0x01000000, 0x7fffffff, 0xff000000]


def fma(a, b, c):
    return float(Decimal(a) * Decimal(b) + Decimal(c))


def words():
    rng = random.Random(1)
    return EDGES + [rng.getrandbits(32) for _ in range(1500)] + [2**32 - 1 - rng.getrandbits(20) for _ in range(500)] + \
        [rng.getrandbits(rng.randint(1, 31)) for _ in range(500)]


def test_neg2_log():
    logs, exps = bm.log_table(), bm.exponent_table()
    for w in words():
        bits = bm._bits(float(2 * w + 1))
        tmp = bits - bm._bits(bm.OFF)
        i, k = (tmp >> 45) & 127, tmp >> 52
        assert 0 <= k <= 33
        inv, lc = logs[i]
        s = fma(bm._float(bits - (k << 52)), inv, 2.0)
        q = 1 / 448.0
        for c in (1 / 192.0, 1 / 80.0, 1 / 32.0, 1 / 12.0, 0.25):
            q = fma(q, s, c)
        got = (exps[k] + lc) + fma(s * s, q, s)
        ref = -2 * (Decimal(2 * w + 1) / 2**33).ln()
        assert abs(Decimal(got) - ref) < 3 * U * ref, w


def test_cos_sin():
    sectors = bm.sector_table()
    for w in words():
        d = float(2 * (w & 0xffffff) + 1 - (1 << 24)) * 7.31459039633579843e-10
        d2 = d * d
        sd = fma(d2 * d, fma(d2, 1 / 120.0, -1 / 6.0), d)
        c1 = d2 * fma(d2, fma(d2, -1 / 720.0, 1 / 24.0), -0.5)
        c, s = sectors[w >> 24]
        rc, rs = bm.cossin(2 * bm.PI * ((Decimal(w) + Decimal("0.5")) / 2**32) - bm.PI)
        assert abs(Decimal(c + fma(-s, sd, c * c1)) - rc) < 2 * U and abs(Decimal(s + fma(c, sd, s * c1)) - rs) < 2 * U
