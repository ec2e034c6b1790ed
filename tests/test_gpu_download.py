"""Results that leave the device through the staging buffers (upload.cpp): blocks and
generators around the sizes where a copy is staged, into pageable and pinned arrays, and
long sequences transposed on the device."""
import numpy as np
import pytest
import torch

import rust_rank_b200 as rr
from rust_rank_b200 import synth

pytestmark = pytest.mark.gpu

P = 2013265921


@pytest.mark.parametrize("n", [1 << 16, (1 << 16) + 7, 700_001])
def test_block_round_trip(ctx, n):
    """With no application queued the block is the caller's, whatever the size (the copies are
    staged from 4 MB on, in pieces of 2 MB); pinned and pageable targets agree."""
    b = 16
    V = synth.random_vectors(b, n, P, 1)
    a = rr.CsrMatrix.from_arrays(np.array([0, 1], np.int64), [0], [1], 1, n)
    dr, dc = synth.preconditioners(1, n, P, 2)
    ks = rr.KrylovStream(a.to_device(P, ctx), V, dr, dc, 0)
    assert np.array_equal(ks.get_curv(), V)
    pinned = torch.empty((b, n), dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    assert np.array_equal(ks.get_curv(pinned), V)
    ks.close()


@pytest.mark.parametrize("terms", [1022, 1024, 1300, 4096])
@pytest.mark.parametrize("b", [1, 5, 16])
def test_long_fetch_equals_short_ones(ctx, b, terms):
    rowptr, col, val, m, n = synth.incidence_fast(120, 100, 3, 8, 0, P, 4)
    dr, dc = synth.preconditioners(m, n, P, 5)
    V = synth.random_vectors(b, n, P, 6)
    ks = rr.KrylovStream(rr.CsrMatrix.from_arrays(rowptr, col, val, m, n).to_device(P, ctx), V, dr, dc, 0)
    ks.step_device(terms // 2)
    total = 2 * (terms // 2) + 1
    whole = np.full((b * (b + 1) // 2, total + 3), 7, np.uint32)
    ks.fetch(0, total, whole)
    parts = np.full_like(whole, 7)
    for lo in range(0, total, 300):
        ks.fetch(lo, min(lo + 300, total), parts)
    assert np.array_equal(whole, parts)
    ks.close()
