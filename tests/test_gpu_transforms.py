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
