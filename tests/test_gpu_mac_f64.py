"""GPU tests of the key-switch MAC on the FP64 pipe (csrc/mac_f64.cuh):
equal to the CUDA-core MAC word for word, and to the oracle on sampled pairs."""
import numpy as np
import pytest

import ckks_b200 as cb
from ckks_b200.params import chain

pytestmark = pytest.mark.gpu


def setup(log_n, q_bits, p_bits, n_ct, steps, base_log, seed, plant=False):
    q, p = chain(1 << log_n, q_bits, p_bits)
    ctx = cb.Context(log_n, q, p)
    n = ctx.n
    rng = np.random.default_rng(seed)
    s = rng.integers(-1, 2, n).astype(np.int8)
    ks = [ctx.rotation_exponent_left(r) for r in steps]
    keys = [cb.KeySwitchKey.hybrid_generate(ctx, len(q), base_log, k, s, seed=seed + i) for i, k in enumerate(ks)]
    cts = np.stack([np.stack([rng.integers(0, m, (2, n), dtype=np.uint64) for m in q], axis=1) for _ in range(n_ct)])
    if plant:  # a parts whose balanced digits contain -B/2: the carry corrections
        Q = int(np.prod([int(m) for m in q], dtype=object))
        for c in range(0, n, 5):
            v = (Q - (1 << (base_log - 1)) * (1 + (c % 3) * (1 << base_log))) % Q
            cts[0, 1, :, c] = [v % m for m in q]
    return q, p, ctx, ks, keys, cts


# pieces of two and of three (60-bit limbs in Q), one key (two components a thread), one
# ciphertext, partial ciphertext and key groups, several key chunks, the smallest ring,
# digit counts odd and beyond two folds (base 2^8: 38 digits), 160 pairs exactly
@pytest.mark.parametrize("log_n,q_bits,p_bits,n_ct,n_keys,base_log,plant", [
    (4, (30,) * 3, (31,), 5, 4, 8, False),
    (10, (50,) * 3, (60,), 1, 1, 32, True),
    (10, (50,) * 6, (60, 60), 16, 10, 8, False),
    (10, (60, 40, 40), (60,), 7, 3, 20, True),
    (11, (50,) * 4, (60,) * 3, 13, 9, 32, True),
    (10, (55,) * 2, (61,), 2, 17, 32, False),
    (12, (50,) * 9, (60,), 3, 6, 8, False),
])
def test_f64_mac_equals_cuda_core_mac(oracle, cuda, log_n, q_bits, p_bits, n_ct, n_keys, base_log, plant):
    q, p, ctx, ks, keys, cts = setup(log_n, q_bits, p_bits, n_ct, range(1, n_keys + 1), base_log, 31 + n_ct, plant)
    d = cb.as_u64_tensor(cts)
    got = cb.to_numpy_u64(cb.rotate_hoisted(ctx, keys, d))
    assert ctx.last_mac_path == "fp64"
    ctx.tensor_cores = False
    assert np.array_equal(got, cb.to_numpy_u64(cb.rotate_hoisted(ctx, keys, d)))
    assert ctx.last_mac_path == "cuda_cores"
    for c, g in {(0, 0), (n_ct - 1, n_keys - 1)}:
        want = oracle.hybrid_rotate(q, p, keys[g].download(), ks[g], base_log, cts[c])
        assert np.array_equal(got[c, g], want), (c, g)


# groups on both sides of the line: it follows the primes' width, the digits, the keys begun and
# the carry corrections to expect
@pytest.mark.parametrize("q_bits,n_ct,n_keys,base_log,path", [
    ((60,) * 6, 16, 8, 32, "fp64"), ((60,) * 6, 16, 9, 32, "tensor_cores"), ((60,) * 6, 5, 24, 32, "tensor_cores"),
    ((60,) * 6, 16, 9, 20, "fp64"), ((50,) * 6, 16, 9, 32, "fp64"), ((50,) * 20, 16, 9, 36, "tensor_cores"),
    ((50,) * 6, 1, 33, 32, "fp64"),
])
def test_faster_mac_by_width_digits_and_keys(cuda, q_bits, n_ct, n_keys, base_log, path):
    q, p, ctx, ks, keys, cts = setup(12, q_bits, (60,), n_ct, range(1, n_keys + 1), base_log, 17)
    d = cb.as_u64_tensor(cts)
    got = cb.to_numpy_u64(cb.rotate_hoisted(ctx, keys, d))
    assert ctx.last_mac_path == path
    ctx.tensor_cores = False
    assert np.array_equal(got, cb.to_numpy_u64(cb.rotate_hoisted(ctx, keys, d)))


def test_tensor_core_mac_corrections_in_a_full_group(cuda):
    """16 x 18 pairs stay on the tensor-core MAC: its carry corrections against the CUDA-core MAC's."""
    q, p, ctx, ks, keys, cts = setup(12, (50,) * 4, (60,), 16, range(1, 19), 32, 91, plant=True)
    d = cb.as_u64_tensor(cts)
    got = cb.to_numpy_u64(cb.rotate_hoisted(ctx, keys, d))
    assert ctx.last_mac_path == "tensor_cores"
    ctx.tensor_cores = False
    assert np.array_equal(got, cb.to_numpy_u64(cb.rotate_hoisted(ctx, keys, d)))


def test_two_piece_sums_at_their_bound(oracle, cuda):
    """A ciphertext of one constant whose base-2^25 digits all lie just above -2^24 and an uploaded
    key whose words' low pieces do: over 57 digits the unit sums grow with one sign through two
    full folds, and the centred high-piece sums of some slots with them."""
    q, p = chain(1 << 8, (50,) * 29, (60,))
    ctx = cb.Context(8, q, p)
    n, base_log = ctx.n, 25
    rng = np.random.default_rng(25)
    k = ctx.rotation_exponent_left(1)
    shape = (cb.KeySwitchKey.hybrid_generate(ctx, len(q), base_log, k, np.ones(n, np.int8), seed=1).info()[0],
             len(q) + 1, 2, n)
    entries = np.empty(shape, np.uint64)
    for i, m in enumerate(q + p):
        high = rng.integers(0, int(m) >> 26, (shape[0], 2, n), dtype=np.int64)
        entries[:, i] = ((high << 25) - (1 << 24) + rng.integers(0, 1 << 8, high.shape)) % int(m)
    key = cb.KeySwitchKey.hybrid_upload(ctx, len(q), base_log, k, entries)
    value = sum((-(1 << 24) + 1 + 2 * int(r)) << (base_log * j) for j, r in enumerate(rng.integers(0, 1 << 7, 57)))
    ct = np.zeros((1, 2, len(q), n), np.uint64)
    ct[0, 1, :, 0] = [value % int(m) for m in q]
    d = cb.as_u64_tensor(ct)
    got = cb.to_numpy_u64(cb.rotate_hoisted(ctx, [key], d))
    assert ctx.last_mac_path == "fp64"
    ctx.tensor_cores = False
    assert np.array_equal(got, cb.to_numpy_u64(cb.rotate_hoisted(ctx, [key], d)))
    assert ctx.last_mac_path == "cuda_cores"
    assert np.array_equal(got[0, 0], oracle.hybrid_rotate(q, p, entries, k, base_log, ct[0]))
