"""CPU tests of the bounds behind the column CRT (csrc/gadget.cu, crt_columns): sums of signed
25-bit products stay exact doubles for a run of limbs, a carry pass brings every column to
[-2^24, 2^24], and the double quotient leaves the sign open only within 2^-40 of a half."""
import random

import numpy as np


def test_runs_stay_exact():
    for run, pieces in ((14, 2), (9, 3)):
        carried = 1 << 29  # a carried column with what the one below hands up
        assert run * pieces * (1 << 48) + carried < 1 << 53


def test_carry_pass():
    rng = random.Random(3)
    big = 6755399441055744.0 * 33554432.0
    for _ in range(300):
        acc = [float(rng.randrange(-(1 << 53), 1 << 53)) for _ in range(8)]
        total = sum(int(a) << (25 * c) for c, a in enumerate(acc))
        for c in range(7):
            hi = (acc[c] + big) - big
            assert int(hi) % (1 << 25) == 0
            acc[c] -= hi
            acc[c + 1] += hi / 33554432.0
            assert abs(acc[c]) <= 1 << 24
        assert sum(int(a) << (25 * c) for c, a in enumerate(acc)) == total


def test_quotient_sum_error():
    """64 centred fractions: every rounding is at most half an ulp of 32, with the reciprocal's."""
    rng = random.Random(5)
    from fractions import Fraction
    for _ in range(200):
        f, exact = np.float64(0), Fraction(0)
        for _ in range(64):
            q = rng.randrange((1 << 49) + 1, 1 << 50) | 1
            u = rng.randrange(-(q // 2), q // 2 + 1)
            f = f + np.float64(u) * (np.float64(1.0) / np.float64(q))  # one rounding more than the FMA
            exact += Fraction(u, q)
        assert abs(Fraction(float(f)) - exact) < Fraction(1, 1 << 41)
