"""Fetches of narrow blocks around the lengths from which the terms are transposed on the device
(1024 terms and 6144 words): whole and in pieces, bit-exact against the oracle."""
import numpy as np
import pytest

import oracle
import rust_rank_b200 as rr
from rust_rank_b200 import synth

pytestmark = pytest.mark.gpu

P = 2013265921


@pytest.mark.parametrize("b,lengths", [(1, (1023, 1025, 6143, 6144)), (2, (1024, 2047, 2048)), (3, (1023, 1024)),
                                       (4, (614, 1024))])
def test_narrow_fetches(ctx, b, lengths):
    rowptr, col, val, m, n = synth.incidence_fast(40, 30, 3, 8, 0, P, 4)
    dr, dc = synth.preconditioners(m, n, P, 5)
    V = synth.random_vectors(b, n, P, 6)
    dm = rr.CsrMatrix.from_arrays(rowptr, col, val, m, n).to_device(P, ctx)
    ks = rr.KrylovStream(dm, V, dr, dc, 0)
    total = 2 * (max(lengths) // 2) + 3
    ks.step_device(total // 2)
    ref, _, _ = oracle.krylov(rowptr, col, val, m, n, P, dr, dc, V, 0, total - 1)
    for count in lengths:
        for lo in (0, total - count):
            seq = np.full((b * (b + 1) // 2, total + 1), 7, np.uint32)
            ks.fetch(lo, lo + count, seq)
            assert np.array_equal(seq[:, lo : lo + count], ref[:, lo : lo + count])
            assert (seq[:, :lo] == 7).all() and (seq[:, lo + count :] == 7).all()
    ks.close()
    dm.close()
