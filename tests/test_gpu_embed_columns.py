"""GPU test of the embedding's column stages (csrc/embed.cu, k_dit_cols) at every ring degree
they run for, one and several messages, and of the encoder's reduction for narrow and wide
primes: every residue and every double against the oracle."""
import numpy as np
import pytest

import ckks_b200 as cb
from ckks_b200.params import chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,messages", [(11, 3), (13, 1), (14, 2), (15, 1), (17, 1)])
def test_encode_and_decode(oracle, cuda, log_n, messages):
    q, _ = chain(1 << log_n, (61, 30, 50))
    ctx = cb.Context(log_n, q)
    rng = np.random.default_rng(log_n)
    z = rng.normal(size=(messages, ctx.n // 2)) + 1j * rng.normal(size=(messages, ctx.n // 2))
    z[0, :4] = [0, 2.0 ** 12, -2.0 ** 12, 1j]
    poly = cb.encode(ctx, z, len(q), 2.0 ** 50)
    back = cb.decode(ctx, poly, 2.0 ** 50).cpu().numpy()
    for i in range(messages):
        want = oracle.encode(z[i], q, 2.0 ** 50)
        assert np.array_equal(cb.to_numpy_u64(poly[i]), want), i
        assert np.array_equal(back[i].view(np.float64), oracle.decode(q, want, 2.0 ** 50).view(np.float64)), i
