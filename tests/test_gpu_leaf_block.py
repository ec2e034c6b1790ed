"""Leaf blocks of the PM-basis (pmleaf.cu) at the edges of their variants, bit-exact
against the oracle: every column-count variant (n <= 4, 8, 16, 32), blocks of one to
the largest number of leaves, and tiny primes, where pivots away from the front of the
column list and rows without a pivot are common."""
import numpy as np
import pytest

import oracle
import rust_rank_b200 as rr

pytestmark = pytest.mark.gpu

CASES = [(1, 64), (1, 128), (2, 1), (3, 2), (4, 64), (5, 4), (7, 32), (8, 128), (9, 32), (11, 16), (15, 64), (16, 2),
         (16, 32), (17, 16), (20, 32), (24, 8), (31, 4), (32, 1), (32, 16)]


@pytest.mark.parametrize("p", [3, 7, 101, 2147483647])
@pytest.mark.parametrize("b,d", CASES)
def test_leaf_block_matches_oracle(ctx, b, d, p):
    rng = np.random.default_rng(1000 * b + d + p % 997)
    np_ = b * (b + 1) // 2
    seqs = [rng.integers(0, p, size=(np_, d + 1)).astype(np.uint32)]
    # entries of rank about half: zero rows and columns in the residuals
    sparse = seqs[0] * (rng.random((np_, 1)) < 0.4)
    seqs.append(np.ascontiguousarray(sparse.astype(np.uint32)))
    for seq, (M, delta) in zip(seqs, rr.PM_Basis_batch(seqs, d, p, ctx)):
        Mo, do = oracle.pm_basis(seq, b, d, p)
        assert np.array_equal(M, Mo.astype(np.uint32))
        assert np.array_equal(delta, do)
