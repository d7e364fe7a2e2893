"""The residue-system form of the tensor-core Park product (csrc/park.cu, namespace rns),
restated on the CPU: the number of moduli, the quotient k from 2^27-scaled reciprocals and
the final combination give the exact product modulo q, at the extremes of the sums too."""
import math
import os
import random
import re

import pytest

MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193, 191, 181, 179, 173]


def moduli_for(inner, q):
    need = 1.05 + math.log2(inner) + 2.0 * math.log2(q - 1)
    have = 0.0
    for n, m in enumerate(MODULI):
        have += math.log2(m)
        if have > need:
            return n + 1
    return 0


def combine(w, mods, q):
    """k_rns_combine for one output, with its word sizes checked."""
    M = math.prod(mods)
    s = sum(wi * ((1 << 27) // m) for wi, m in zip(w, mods))
    assert s + 8192 < 1 << 32
    k = (s + 8192) >> 27
    nm = (-M) % q
    lo = sum(wi * ((M // m % q) & 0xFFFFFFFF) for wi, m in zip(w, mods)) + k * (nm & 0xFFFFFFFF)
    hi = sum(wi * ((M // m % q) >> 32) for wi, m in zip(w, mods)) + k * (nm >> 32)
    assert lo < 1 << 45 and hi < 1 << 45 and 2 * q + lo < 1 << 64
    return k, (lo + (hi << 32)) % q


def test_one_list_of_moduli():
    """The kernels', the bench's and this file's."""
    root = os.path.join(os.path.dirname(__file__), "..")
    for path, name in (("ccmm-rs_b200/csrc/park.cu", r"kModuli\[kMaxMod\] = \{"), ("bench.py", r"PARK_MODULI = \(")):
        text = open(os.path.join(root, path)).read()
        assert [int(x) for x in re.search(name + r"([\d,\s]+)[})]", text).group(1).split(",")] == MODULI, path


def test_moduli_are_coprime_bytes():
    for i, a in enumerate(MODULI):
        assert 2 <= a <= 256
        for b in MODULI[:i]:
            assert math.gcd(a, b) == 1


@pytest.mark.parametrize("q", [(1 << 24) + 1, 0x7ffff6001, (1 << 47) - 115, 0xfffffffffffc001, (1 << 62) - 57])
@pytest.mark.parametrize("inner", [1, 2, 4096, 33024])
def test_exact_for_every_sum(q, inner):
    n = moduli_for(inner, q)
    assert n, "enough moduli up to 2^62 and the longest inner sum"
    assert inner * 255 * 255 < 1 << 31
    mods = MODULI[:n]
    M = math.prod(mods)
    top = inner * (q - 1) ** 2
    assert 2 * top < M
    rng = random.Random(q + inner)
    for x in [0, 1, top, top - 1, q - 1, q, (q - 1) ** 2] + [rng.randrange(top + 1) for _ in range(300)]:
        if x > top:
            continue
        w = [x * pow(M // m, -1, m) % m for m in mods]
        k, got = combine(w, mods, q)
        assert x == sum(wi * (M // m) for wi, m in zip(w, mods)) - k * M
        assert got == x % q


def test_reductions_are_exact():
    rng = random.Random(1)
    for m in MODULI:
        small, floor = -(-(1 << 32) // m), (1 << 32) // m
        for s in [0, m - 1, m, 8 * 255 * 255] + [rng.randrange(8 * 255 * 255 + 1) for _ in range(200)]:
            assert s - ((s * small) >> 32) * m == s % m
        for s in [0, m - 1, m, (1 << 31) - 1] + [rng.randrange(1 << 31) for _ in range(200)]:
            r = s - ((s * floor) >> 32) * m
            assert (r - m if r >= m else r) == s % m
