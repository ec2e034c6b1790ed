"""Transforms of the PM-basis products at the edges of their passes: even and odd numbers of
stages, several polynomials per CTA, the longest in shared memory and the first with stages in
global memory, over the matrix prime and over the CRT primes -- bit-exact against the oracle."""
import numpy as np
import pytest

import oracle
import rust_rank_b200 as rr

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[True, False], ids=["tensor", "cuda-core"])
def pm_ctx(request):
    c = rr.Context(0)
    c.set_pm_tensor_cores(request.param)
    yield c
    c.close()


@pytest.mark.parametrize("p", [3323, 2013265921])
@pytest.mark.parametrize("b,d", [(1, 2), (1, 4), (1, 8), (1, 16), (1, 64), (1, 128), (2, 512), (1, 2048), (1, 4096), (1, 8192),
                                 (2, 16384)])
def test_lengths(pm_ctx, b, d, p):
    rng = np.random.default_rng(b + d)
    seq = rng.integers(0, p, size=(b * (b + 1) // 2, d + 1)).astype(np.uint32)
    M, delta = rr.PM_Basis(seq, d, p, pm_ctx)
    Mo, do = oracle.pm_basis(seq, b, d, p)
    assert np.array_equal(M, Mo.astype(np.uint32))
    assert np.array_equal(delta, do)


@pytest.mark.parametrize("b,d,nb", [(8, 512, 7), (8, 512, 8), (13, 256, 5), (16, 128, 4), (32, 64, 2)])
def test_batches_around_the_direct_products(ctx, b, d, nb):
    """Batches on both sides of 128 rows, from which the shorter products are transforms too."""
    p = 2013265921
    rng = np.random.default_rng(nb)
    seqs = [rng.integers(0, p, size=(b * (b + 1) // 2, d + 1)).astype(np.uint32) for _ in range(nb)]
    for seq, (M, delta) in zip(seqs, rr.PM_Basis_batch(seqs, d, p, ctx)):
        Mo, do = oracle.pm_basis(seq, b, d, p)
        assert np.array_equal(M, Mo.astype(np.uint32)) and np.array_equal(delta, do)
