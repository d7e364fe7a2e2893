"""The two-piece sums of the FP64 key-switch MAC (csrc/mac_f64.cuh, k_mac_f64<2, ..>), restated
on the CPU operation for operation: s00, s01 and s11 in units of 1, 2^25 and 2^50, folded every
kFold terms (s01) and 2 kFold terms (s00, s11). Every sum must be an exact double, an integer of
at most 2^53 units, for any words of a prime below 2^50, and the residue the exact one."""
import os
import random
import re

import pytest

SRC = os.path.join(os.path.dirname(__file__), "..", "ccmm-rs_b200", "csrc", "mac_f64.cuh")
FOLD = int(re.search(r"constexpr int kFold = (\d+);", open(SRC).read()).group(1))
STAGE = int(re.search(r"constexpr int kJs = (\d+);", open(SRC).read()).group(1))
TOP = 1 << 53
PRIMES = [0x3ffffffd20001, (1 << 50) - (1 << 17) * 23 + 1, (1 << 49) + 9, (1 << 40) - 87, (1 << 30) + 3]


def split(x, q):
    """x0 in [-2^24, 2^24) and x1 in units of 2^25, of the centred word."""
    c = (x - q if x > q >> 1 else x) + (1 << 24)
    return (c & ((1 << 25) - 1)) - (1 << 24), c >> 25


def exact(v):
    assert abs(v) <= TOP, "sum beyond an exact double: 2^48 times %.4f" % (abs(v) / 2.0 ** 48)
    return v


def center(v, q):
    """nttf::center of the integer v (a double): v - rint(v fl(1/q)) q."""
    t = round(float(v) * (1.0 / float(q)))  # both round half to even; t is below 2^53
    r = v - t * q
    assert abs(r) < TOP
    return r


def mac(ys, ks, q):
    s00 = s01 = s11 = 0
    every = False
    for j, (y, k) in enumerate(zip(ys, ks)):
        if j and j % FOLD == 0:
            s00 = exact(s00 + center(s01 << 25, q))
            s01 = 0
            if every:
                s00 = center(s00, q)
                s00 = center(exact(s00 + center(s11 << 50, q)), q)
                s11 = 0
            every = not every
        (y0, y1), (k0, k1) = split(y, q), split(k, q)
        s01 = exact(s01 + y0 * k1)
        s00 = exact(s00 + y0 * k0)
        s11 = exact(s11 + y1 * k1)
        s01 = exact(s01 + y1 * k0)
    m = exact(center(s01 << 25, q) + center(s11 << 50, q))
    return exact(center(s00, q) + m) % q


def test_unit_bound():
    """s00 in units of 2^48: a centred start, kFold terms twice, a centred s01 at each fold. A
    centred value is q/2 < 2^49 and a rounding of the quotient (below 2^26 for s01)."""
    assert FOLD % STAGE == 0
    centred = (1 << 49) + (1 << 26)
    assert 2 * FOLD * (1 << 48) + 3 * centred <= TOP
    assert 2 * FOLD * (1 << 48) <= TOP  # s01 takes two products a term, s11 one for 2 kFold terms


@pytest.mark.parametrize("q", PRIMES)
@pytest.mark.parametrize("digits", [FOLD, 2 * FOLD, 2 * FOLD + 1, 57, 61, 113])
def test_extreme_words_are_exact(q, digits):
    rng = random.Random(q + digits)
    for trial in range(60):
        sign = rng.choice([-1, 1])

        def word(s):  # low piece near its bound, any high piece
            low = -(1 << 24) + rng.randrange(1 << 8) if s < 0 else (1 << 24) - 1 - rng.randrange(1 << 8)
            return ((rng.randrange(q >> 25) << 25) + low) % q if q >> 26 else rng.randrange(q)
        ys, ks = [word(sign) for _ in range(digits)], [word(sign) for _ in range(digits)]
        if trial % 3 == 2:
            ys, ks = [rng.randrange(q) for _ in ys], [q >> 1] * digits
        assert mac(ys, ks, q) == sum(y * k for y, k in zip(ys, ks)) % q


def test_sums_that_the_folds_bring_to_their_bound():
    """Low pieces of one sign, the last high piece of every run chosen so that its centred s01 is
    near q/2 as well, so s00 comes close to the bound of test_unit_bound."""
    q = PRIMES[0]
    rng = random.Random(1)
    y = q - (1 << 24)
    for trial in range(40):
        ks = []
        while len(ks) < 61:
            run = min(FOLD, 61 - len(ks))
            highs = [rng.randrange(q >> 26) for _ in range(run - 1)]
            highs.append(max((rng.randrange(q >> 26) for _ in range(1000)),
                             key=lambda h: center(-(sum(highs) + h) << 49, q)))
            ks += [((h << 25) - (1 << 24) + rng.randrange(1 << 8)) % q for h in highs]
        ys = [y + rng.randrange(1 << 8) for _ in ks]
        assert mac(ys, ks, q) == sum(a * b for a, b in zip(ys, ks)) % q
