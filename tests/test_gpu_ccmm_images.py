"""GPU test of the CCMM slot products' A images and epilogue (csrc/ccmm_tc.cu) at their edges:
row counts around 8 and 32, odd inner sizes, and primes on both sides of 2^50 (the plane
combination on the FP64 pipe and the integer one), against the CUDA-core products."""
import numpy as np
import pytest

import ckks_b200 as cb
from ckks_b200.params import chain

pytestmark = pytest.mark.gpu


def compare(ctx, key, q, m, k, n):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + k + n)

    def matrix(*lead):
        x = torch.empty(lead + (2, len(q), ctx.n), dtype=torch.int64, device="cuda")
        for i, mod in enumerate(q):
            x[..., i, :].random_(0, mod, generator=gen)
            x[0, 0, :, i, :4] = mod - 1
        return x

    a, b = matrix(k, m), matrix(n, k)
    got = cb.matmul_structured(ctx, key, a, b, m, k, n)
    torch.cuda.synchronize()
    assert ctx.last_mac_path == "tensor_cores"
    ctx.tensor_cores = False
    assert torch.equal(got, cb.matmul_structured(ctx, key, a, b, m, k, n))


@pytest.mark.parametrize("q_bits", [(50, 50), (55, 40), (30, 49)])
@pytest.mark.parametrize("m,k,n", [(7, 1, 2), (8, 3, 17), (9, 9, 1), (31, 2, 3), (32, 5, 33), (33, 64, 2)])
def test_tensor_cores_equal_cuda_cores(cuda, q_bits, m, k, n):
    q, _ = chain(1 << 8, q_bits)
    ctx = cb.Context(8, q)
    key = cb.KeySwitchKey.relin_generate(ctx, len(q), 20, np.random.default_rng(2).integers(-1, 2, ctx.n), seed=5)
    compare(ctx, key, q, m, k, n)


# an A of more than 2^28 words is transformed and written in several calls (60 entries each here):
# whole pairs of inner indices a call, odd inner sizes, rows below 8, fewer entries than a pair
@pytest.mark.parametrize("m,k,n", [(20, 5, 1), (7, 19, 2), (64, 3, 1), (29, 4, 1), (1, 64, 1)])
def test_images_written_in_several_calls(cuda, m, k, n):
    q, _ = chain(1 << 17, (50,) * 17)
    ctx = cb.Context(17, q)
    key = cb.KeySwitchKey.relin_generate(ctx, len(q), 45, np.random.default_rng(2).integers(-1, 2, ctx.n), seed=5)
    compare(ctx, key, q, m, k, n)
