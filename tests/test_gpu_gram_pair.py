"""Both Gram terms of an application formed over the columns of A (krylov.cu): the odd and the
even term bit-exact against the oracle at the edges of the row batches (widths 4 and 8), of the
128-row tiles of the Gram pass (widths 16 and 32) and of the tail of empty columns."""
import numpy as np
import pytest

import oracle
import rust_rank_b200 as rr
from rust_rank_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,used", [(1, 1), (15, 15), (33, 32), (127, 127), (128, 100), (129, 129), (300, 129),
                                    (148 * 128 + 1, 148 * 128 + 1), (148 * 128 * 2 + 130, 148 * 128 + 3)])
@pytest.mark.parametrize("b,p", [(3, 2013265921), (8, 2147483647), (9, 3), (16, 2013265921), (27, 3323), (32, 2147483647)])
def test_both_terms(ctx, n, used, b, p):
    rng = np.random.default_rng(n + b)
    # a row of more than 64 entries keeps the applications on the launched kernels where n allows
    lens = rng.integers(0, min(used, 4) + 1, size=max(n // 2, 3))
    lens[0] = min(used, 70)
    rowptr = np.zeros(len(lens) + 1, np.int64)
    rowptr[1:] = np.cumsum(lens)
    col = np.concatenate([np.sort(rng.choice(used, size=k, replace=False)) for k in lens]).astype(np.int32)
    val = rng.integers(1, p, size=int(rowptr[-1])).astype(np.uint32)
    dr, dc = synth.preconditioners(len(lens), n, p, 5)
    V = synth.random_vectors(b, n, p, 6)
    ks = rr.KrylovStream(rr.CsrMatrix.from_arrays(rowptr, col, val, len(lens), n).to_device(p, ctx), V, dr, dc, 0)
    seq = np.zeros((b * (b + 1) // 2, 7), np.uint32)
    ks.step_device(1)
    ks.step_device(2)
    ks.fetch(0, 7, seq)
    ref, L, cv = oracle.krylov(rowptr, col, val, len(lens), n, p, dr, dc, V, 0, 6)
    assert L == 7
    assert np.array_equal(seq, ref[:, :L])
    assert np.array_equal(ks.get_curv(), cv)
    ks.close()
