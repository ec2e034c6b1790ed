"""The tcgen05 Gram pass (krylov.cu) on blocks of few columns: less than one 128-row tile, where a
column of more than 64 entries keeps the applications off the resident runs at every width."""
import numpy as np
import pytest

import oracle
import rust_rank_b200 as rr
from rust_rank_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 5, 15, 16, 33, 63, 64])
@pytest.mark.parametrize("b,p", [(9, 3323), (16, 2013265921), (16, 2147483647), (24, 3), (32, 2147483647)])
def test_both_terms_of_few_columns(ctx, n, b, p):
    rng = np.random.default_rng(100 * n + b)
    m = 70  # a full first column
    rows = [np.unique(np.concatenate([[0], rng.choice(n, size=min(n, 3))])) for _ in range(m)]
    rowptr = np.zeros(m + 1, np.int64)
    rowptr[1:] = np.cumsum([len(r) for r in rows])
    col = np.concatenate(rows).astype(np.int32)
    val = rng.integers(1, p, size=int(rowptr[-1])).astype(np.uint32)
    dr, dc = synth.preconditioners(m, n, p, 5)
    V = synth.random_vectors(b, n, p, 6)
    dm = rr.CsrMatrix.from_arrays(rowptr, col, val, m, n).to_device(p, ctx)
    ks = rr.KrylovStream(dm, V, dr, dc, 0)
    before = ks.launch_count()
    ks.step_device(1)
    assert ks.launch_count() - before >= 3  # two passes and the Gram pass; a resident run is two launches
    ks.step_device(5)
    seq = np.zeros((b * (b + 1) // 2, 13), np.uint32)
    ks.fetch(0, 13, seq)
    ref, _, cv = oracle.krylov(rowptr, col, val, m, n, p, dr, dc, V, 0, 12)
    assert np.array_equal(seq, ref[:, :13])
    assert np.array_equal(ks.get_curv(), cv)
    ks.close()
    dm.close()
