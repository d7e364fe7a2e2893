"""GPU test of the relinearization pass that takes two digits at once where the second half of
the transform has an odd number of stages (csrc/ntt.cu, k_fwd2_relin): one digit, pairs, and
an odd last digit, at each such split; exact residues against the oracle."""
import numpy as np
import pytest

import ckks_b200 as cb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n", [6, 7, 10, 11, 14, 15])
@pytest.mark.parametrize("primes,base_log", [(1, 55), (1, 30), (2, 35), (2, 25), (3, 17)])
def test_digit_counts(oracle, cuda, log_n, primes, base_log):
    n = 1 << log_n
    q = [int(x) for x in oracle.primes_below_bits(50, n, primes)]
    ctx = cb.Context(log_n, q)
    rng = np.random.default_rng(log_n + base_log)
    s = rng.integers(-1, 2, n).astype(np.int8)
    key_ref = oracle.relin_key(q, s, base_log, seed=3)
    key = cb.KeySwitchKey.relin_upload(ctx, len(q), base_log, key_ref)
    quad = np.stack([np.stack([rng.integers(0, m, (3, n), dtype=np.uint64) for m in q], axis=1) for _ in range(2)])
    got = cb.to_numpy_u64(cb.relinearize(ctx, key, cb.as_u64_tensor(quad)))
    for c in range(2):
        assert np.array_equal(got[c], oracle.relinearize(q, quad[c], key_ref, base_log)), c
