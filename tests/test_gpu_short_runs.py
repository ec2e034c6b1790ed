"""Applications at width 16 on both sides of the entry counts from which one or two of them are
launches instead of a resident run (queue_apps): which way was taken, and the oracle's terms."""
import numpy as np
import pytest

import oracle
import rust_rank_b200 as rr
from rust_rank_b200 import synth

pytestmark = pytest.mark.gpu

P = 2013265921


@pytest.mark.parametrize("m,nnz,shortest", [(50_000, 199_000, 1), (50_000, 201_000, 2), (180_000, 1_090_000, 2),
                                            (180_000, 1_110_000, 3)])
def test_shortest_run(ctx, m, nnz, shortest):
    rng = np.random.default_rng(nnz)
    n = m // 2
    lens = np.full(m, nnz // m)
    lens[: nnz - int(lens.sum())] += 1
    rowptr = np.zeros(m + 1, np.int64)
    rowptr[1:] = np.cumsum(lens)
    # distinct columns of a row, and no column of more than 64 entries
    first = rng.integers(0, n, size=m)
    col = ((np.repeat(first, lens) + 37 * (np.arange(nnz) - np.repeat(rowptr[:-1], lens))) % n).astype(np.int32)
    for i in np.flatnonzero(np.bincount(col, minlength=n) > 64):
        pytest.fail(f"column {i} is too long")
    val = rng.integers(1, P, size=nnz).astype(np.uint32)
    dr, dc = synth.preconditioners(m, n, P, 1)
    b = 16
    V = synth.random_vectors(b, n, P, 2)
    dm = rr.CsrMatrix.from_arrays(rowptr, col, val, m, n).to_device(P, ctx)
    ks = rr.KrylovStream(dm, V, dr, dc, 0)
    done = 0
    for apps in (1, 2, 3):
        before = ks.launch_count()
        ks.step_device(apps)
        done += apps
        assert (ks.launch_count() - before == 2) == (apps >= shortest), apps  # a run and its finish
    seq = np.zeros((b * (b + 1) // 2, 2 * done + 1), np.uint32)
    ks.fetch(0, 2 * done + 1, seq)
    ref, _, cv = oracle.krylov(rowptr, col, val, m, n, P, dr, dc, V, 0, 2 * done)
    assert np.array_equal(seq, ref) and np.array_equal(ks.get_curv(), cv)
    ks.close()
    dm.close()
