"""GPU test of the digit lift of the forward transforms' first pass (csrc/ntt.cu)."""
import numpy as np
import pytest

import ckks_b200 as cb
from ckks_b200.params import chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("base_log", [40, 50, 51, 52, 53, 60])
def test_digit_lift_at_the_prime_size(oracle, cuda, base_log):
    """Digits around the primes' size (50-bit and 60-bit limbs, 30-bit ones far below it): taken
    signed up to 2^(b-1) <= q, reduced above."""
    q, p = chain(1 << 8, (50, 50, 30), (60,))
    ctx = cb.Context(8, q, p)
    rng = np.random.default_rng(7)
    s = rng.integers(-1, 2, ctx.n).astype(np.int8)
    k = ctx.rotation_exponent_left(1)
    key = cb.KeySwitchKey.hybrid_generate(ctx, len(q), base_log, k, s, seed=7)
    cts = np.stack([np.stack([rng.integers(0, m, (2, ctx.n), dtype=np.uint64) for m in q], axis=1) for _ in range(2)])
    got = cb.to_numpy_u64(cb.rotate(ctx, key, cb.as_u64_tensor(cts)))
    for c in range(2):
        want = oracle.hybrid_rotate(q, p, key.download(), k, base_log, cts[c])
        assert np.array_equal(got[c], want), c
