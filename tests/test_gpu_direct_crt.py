"""GPU tests of the direct exact CRT in 25-bit columns (csrc/gadget.cu, crt_columns) under the
gadget decomposition and the decode: every column size and both piece counts, values whose sign
the 64-bit fraction leaves open (around Q/2), around 0 and Q, and random ones, against the oracle."""
import numpy as np
import pytest

import ckks_b200 as cb
from ckks_b200.params import chain

pytestmark = pytest.mark.gpu

BITS = [(30,), (60,), (50,) * 3, (60, 40, 40), (50,) * 7, (50,) * 11, (61,) * 9, (50,) * 15, (50,) * 19, (50,) * 24,
        (61,) * 20, (50,) * 25]


def setup(q_bits):
    q, _ = chain(1 << 8, q_bits)
    ctx = cb.Context(8, q)
    rng = np.random.default_rng(len(q_bits))
    x = np.stack([rng.integers(0, m, ctx.n, dtype=np.uint64) for m in q])
    Q = int(np.prod([int(m) for m in q], dtype=object))
    # the quotient's double sum is off by under 2^-41, and 2^-40 around a half is compared exactly
    u = Q >> 48
    edges = [0, 1, 2, Q - 1, Q - 2, Q // 2, Q // 2 + 1, Q // 2 - 1, Q // 2 + 2]
    edges += [Q // 2 + s * (k * u + e) for k in (1, 16, 127, 128, 255, 256, 257, 4096) for s in (1, -1) for e in (0, 1)]
    for c, v in enumerate(edges):
        x[:, c] = [(v % Q) % m for m in q]
    return q, ctx, x


@pytest.mark.parametrize("q_bits", BITS)
@pytest.mark.parametrize("base_log", [2, 20, 25, 32, 39, 40])
def test_digits(oracle, cuda, q_bits, base_log):
    q, ctx, x = setup(q_bits)
    got = ctx.bounded_decompose(cb.as_u64_tensor(x), base_log).cpu().numpy()
    assert np.array_equal(got, oracle.bounded_decompose(q, x, base_log))


@pytest.mark.parametrize("q_bits", BITS)
def test_decode(oracle, cuda, q_bits):
    q, ctx, x = setup(q_bits)
    scale = 2.0 ** 40
    if sum(q_bits) > 1000:  # values that stay finite as doubles: below 2^900, both signs
        rng = np.random.default_rng(5)
        for c in range(ctx.n):
            v = int.from_bytes(rng.bytes(112), "little") >> int(rng.integers(0, 896))
            x[:, c] = [(v if c % 2 else -v) % m for m in q]
        scale = 2.0 ** 850
    got = cb.decode(ctx, cb.as_u64_tensor(x), scale).cpu().numpy()
    want = oracle.decode(q, x, scale)
    assert np.isfinite(want.view(np.float64)).all()
    assert np.array_equal(got.view(np.float64), want.view(np.float64))
