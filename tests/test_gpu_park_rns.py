"""The residue-system form of the tensor-core Park product at the edges of its rule (moduli
around 2^24, 2^32 and 2^62, inner sums around 33,024 terms), of its tiles (128 rows, 256 columns,
32-deep steps in stages of four) and of its sums (all zeros, all q - 1), against the 192-bit
CUDA-core sums and the oracle."""
import numpy as np
import pytest

import ckks_b200 as cb

pytestmark = pytest.mark.gpu


def check(oracle, a, b, q):
    da, db = cb.as_u64_tensor(a), cb.as_u64_tensor(b)
    got = cb.to_numpy_u64(cb.park_mod_pp_mm(da, db, q, backend="tensor_cores"))
    assert np.array_equal(got, cb.to_numpy_u64(cb.park_mod_pp_mm(da, db, q, backend="cuda_cores")))
    assert np.array_equal(got[:2], oracle.park_mod_pp_mm(a[:2], b, q))


@pytest.mark.parametrize("q", [1 << 24, (1 << 24) + 1, 1 << 32, (1 << 32) + 1, 0x7ffff6001, (1 << 61) - 1, (1 << 62) - 57, 1 << 62])
@pytest.mark.parametrize("shape", [(1, 1, 1), (128, 32, 256), (129, 33, 257), (3, 129, 1030), (300, 161, 5)])
def test_shapes_and_moduli(oracle, cuda, q, shape):
    r, k, c = shape
    rng = np.random.default_rng(r + k + c)
    check(oracle, rng.integers(0, 2**64, (r, k), dtype=np.uint64), rng.integers(0, 2**64, (k, c), dtype=np.uint64), q)


@pytest.mark.parametrize("inner", [33024, 33025])
def test_longest_inner_sums(oracle, cuda, inner):
    q = 0x7ffff6001
    full = np.full((2, inner), q - 1, np.uint64)
    check(oracle, full, np.full((inner, 3), q - 1, np.uint64), q)
    check(oracle, full, np.zeros((inner, 3), np.uint64), q)


def test_four_byte_modulus_above_the_size_line(cuda):
    q, n = (1 << 24) + 43, 1300
    rng = np.random.default_rng(n)
    a, b = (cb.as_u64_tensor(rng.integers(0, q, (n, n), dtype=np.uint64)) for _ in range(2))
    import torch
    assert torch.equal(cb.park_mod_pp_mm(a, b, q, backend="tensor_cores"),
                       cb.park_mod_pp_mm(a, b, q, backend="cuda_cores"))


def random(rows, cols, q, seed):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.empty((rows, cols), dtype=torch.int64, device="cuda").random_(0, q, generator=gen)


def peak_workspace(call):
    """Device bytes that a call takes from the stream-ordered pool at its peak."""
    import torch
    from cuda.bindings import driver, runtime as rt
    torch.cuda.synchronize()
    err, pool = rt.cudaDeviceGetDefaultMemPool(torch.cuda.current_device())
    assert int(err) == 0
    attr = rt.cudaMemPoolAttr
    before = int(rt.cudaMemPoolGetAttribute(pool, attr.cudaMemPoolAttrUsedMemCurrent)[1])
    assert int(rt.cudaMemPoolSetAttribute(pool, attr.cudaMemPoolAttrUsedMemHigh, driver.cuuint64_t(0))[0]) == 0
    out = call()
    torch.cuda.synchronize()
    return out, int(rt.cudaMemPoolGetAttribute(pool, attr.cudaMemPoolAttrUsedMemHigh)[1]) - before


# row slabs, column slabs and both: residues of the whole product beyond 2 GiB
@pytest.mark.parametrize("shape", [(12000, 1030, 11000), (200, 1, 500000), (600, 1, 500000)])
def test_products_beyond_the_workspace_limit_in_slabs(cuda, shape):
    import torch
    q = (1 << 60) - 93
    (r, k, c), limit = shape, 2 << 30
    a, b = random(r, k, q, 1), random(k, c, q, 2)
    got, peak = peak_workspace(lambda: cb.park_mod_pp_mm(a, b, q, backend="tensor_cores"))
    packed = 8 * k * (r + 8 * c)  # of the byte planes, which may be the larger limit
    assert peak < max(limit, 1.2 * packed) + (64 << 20), peak
    assert torch.equal(got, cb.park_mod_pp_mm(a, b, q, backend="cuda_cores"))


# where writing and reading a residue per modulus and output outweighs the products saved
@pytest.mark.parametrize("bits,shape", [(35, (4096, 64, 4096)), (35, (65536, 32, 16)), (47, (20000, 32, 16)),
                                        (56, (20000, 33, 9)), (60, (20000, 32, 16))])
def test_short_inner_sums_take_the_byte_planes(cuda, bits, shape):
    import torch
    q = (1 << bits) - 115
    a, b = random(*shape[:2], q, 3), random(*shape[1:], q, 4)
    got, peak = peak_workspace(lambda: cb.park_mod_pp_mm(a, b, q, backend="tensor_cores"))
    assert peak < 8 * shape[0] * max(shape[2], 256)  # the residue form takes at least 11 bytes an output
    assert torch.equal(got, cb.park_mod_pp_mm(a, b, q, backend="cuda_cores"))


@pytest.mark.parametrize("bits", [40, 47, 56, 61])  # five to eight bytes
def test_chunked_byte_planes_of_wide_moduli(oracle, cuda, bits):
    """Inner sums beyond the residue system's: several plane launches that add their residues."""
    rng = np.random.default_rng(bits)
    check(oracle, rng.integers(0, 2**64, (3, 33100), dtype=np.uint64), rng.integers(0, 2**64, (33100, 5), dtype=np.uint64),
          (1 << bits) - 115)
