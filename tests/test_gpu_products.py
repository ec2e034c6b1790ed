"""Products above the leaf blocks of the PM-basis at the edges of their dispatch: the longest
direct product, the first transform level, and the CRT primes, for every inner-dimension
variant -- bit-exact against the oracle."""
import numpy as np
import pytest

import oracle
import rust_rank_b200 as rr

pytestmark = pytest.mark.gpu

# (b, d): levels of half length d / 2, d / 4, ... above the block; the direct product takes
# half lengths up to 128 (2b <= 16), 64 (2b <= 32) and 32 (2b <= 64)
CASES = [(1, 256), (1, 1024), (3, 512), (4, 256), (8, 512), (9, 64), (11, 128), (16, 128), (16, 256), (17, 64),
         (24, 128), (32, 32), (32, 128)]


@pytest.mark.parametrize("p", [3323, 2013265921, 2147483647])
@pytest.mark.parametrize("b,d", CASES)
def test_products_match_oracle(ctx, b, d, p):
    rng = np.random.default_rng(b + d)
    seq = rng.integers(0, p, size=(b * (b + 1) // 2, d + 1)).astype(np.uint32)
    M, delta = rr.PM_Basis(seq, d, p, ctx)
    Mo, do = oracle.pm_basis(seq, b, d, p)
    assert np.array_equal(M, Mo.astype(np.uint32))
    assert np.array_equal(delta, do)


@pytest.mark.parametrize("b,d", [(4, 512), (16, 256), (32, 128)])
def test_batched_products(ctx, b, d):
    p = 2013265921
    rng = np.random.default_rng(7)
    seqs = [rng.integers(0, p, size=(b * (b + 1) // 2, d + 1)).astype(np.uint32) for _ in range(3)]
    for seq, (M, delta) in zip(seqs, rr.PM_Basis_batch(seqs, d, p, ctx)):
        M1, d1 = rr.PM_Basis(seq, d, p, ctx)
        assert np.array_equal(M, M1) and np.array_equal(delta, d1)
