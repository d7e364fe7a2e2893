"""CPU tests: the FP64 twist multiplication whose quotient factor is formed on the
fly (csrc/ntt.cu: mulmod with wp = fl(w fl(1/q)) instead of fl(w/q)), and the bounds
that the two halves of a transform then keep.

wp differs from w/q by at most 2^-53 (1/q rounded) + 2^-54 (the product rounded,
wp < 1), and fl(Y wp) by half an ulp more, so with t = rint(fl(Y wp))
  |Y w - t q| <= (1/2 + 1.5 |Y| 2^-53 + ulp(|Y|) / 2) q:
below 2 q for |Y| < 4.5 q (forward, q < 2^50) and below 3 q for |Y| < 2^53 (inverse).
"""
import random
from fractions import Fraction

PRIMES = [(1 << 50) - (1 << 17) * 23 + 1, 0x3ffffffd20001, (1 << 40) - 87, (1 << 30) + 3]


def mulmod_twist(y, w, q):
    wp = float(Fraction(float(w)) * Fraction(1.0 / float(q)))
    t = round(float(Fraction(y) * Fraction(wp)))
    h = float(y * w)
    r = y * w - t * q
    low = y * w - int(h)
    assert abs(low) < 1 << 53 and abs(int(h) - t * q) < 1 << 53  # both parts are exact doubles
    return r


def test_twist_bounds():
    rng = random.Random(4)
    for q in PRIMES:
        for lim, bound in ((int(4.5 * q), 2), (min((1 << 53) - 1, 8 * q), 3)):
            for k in range(4000):
                y = rng.choice([lim - 1, lim - rng.randrange(1 << 20), rng.randrange(lim)]) * rng.choice([1, -1])
                w = rng.choice([q - 1, q - 2, rng.randrange(q), rng.randrange(q)])
                r = mulmod_twist(y, w, q)
                assert (r - y * w) % q == 0 and abs(r) < bound * q, (q, y, w, r)


def test_forward_half_from_twisted_inputs_stays_below_2_53():
    """A stage adds |r| <= band(bound) q (test_f64_bounds_cpu): four stages from 2 q."""
    q = 1 << 50
    b = 2.0
    for _ in range(4):
        b += 0.75 if b * q < 1 << 51 else 1.0 if b * q < 1 << 52 else 1.5
    assert b * q < 1 << 53


def test_signed_digits_need_no_reduction():
    """Digits in [-2^(b-1), 2^(b-1)) with 2^(b-1) <= q enter the network as they are: the
    bits 0x4338.. + d are the double 2^52 + 2^51 + d for |d| <= 2^51 (d = 2^51 excluded)."""
    import struct
    for d in (0, 1, -1, (1 << 31) - 1, -(1 << 31), (1 << 51) - 1, -(1 << 51)):
        bits = (0x4338000000000000 + d) & (2**64 - 1)
        x = struct.unpack("<d", struct.pack("<Q", bits))[0]
        assert x - 6755399441055744.0 == d
