"""Runs of applications with the CSR in shared memory (resident.cu): bit-exact against the
oracle at the edges of their row batches, degrees and run lengths, and side by side with
other runs on the device."""
import threading

import numpy as np
import pytest

import oracle
import rust_rank_b200 as rr
from rust_rank_b200 import synth

pytestmark = pytest.mark.gpu

P = 2013265921


def _csr(lens, n, p, seed):
    """Rows of the given lengths, distinct random columns, values in [1, p)."""
    rng = np.random.default_rng(seed)
    rowptr = np.zeros(len(lens) + 1, np.int64)
    rowptr[1:] = np.cumsum(lens)
    col = np.concatenate([np.sort(rng.choice(n, size=k, replace=False)) for k in lens] + [np.zeros(0, np.int64)])
    val = rng.integers(1, p, size=int(rowptr[-1]))
    return rowptr, col.astype(np.int32), val.astype(np.uint32), len(lens), n


def _check(ctx, mat, b, p, apps, seed=3):
    rowptr, col, val, m, n = mat
    dr, dc = synth.preconditioners(m, n, p, seed)
    V = synth.random_vectors(b, n, p, seed + 1)
    ks = rr.KrylovStream(rr.CsrMatrix.from_arrays(rowptr, col, val, m, n).to_device(p, ctx), V, dr, dc, 0)
    total = sum(apps)
    seq = np.zeros((b * (b + 1) // 2, 2 * total + 1), np.uint32)
    done = 0
    for k in apps:
        ks.step_device(k)
        done += k
    ks.fetch(0, 2 * total + 1, seq)
    ref, L, cv = oracle.krylov(rowptr, col, val, m, n, p, dr, dc, V, 0, 2 * total)
    assert L == 2 * total + 1
    assert np.array_equal(seq, ref[:, :L])
    assert np.array_equal(ks.get_curv(), cv)
    ks.close()


@pytest.mark.parametrize("p", [3, 3323, P, 2147483647])
@pytest.mark.parametrize("b", [1, 4, 5, 8, 9, 16])
def test_degrees_and_row_batches(ctx, b, p):
    """Row counts around a row batch, empty rows, rows of up to 64 entries (the longest the
    run takes) in both directions, and of 65, which take the pass kernels."""
    rng = np.random.default_rng(b)
    for m, n, top in ((1, 1, 1), (33, 70, 64), (64, 31, 7), (700, 500, 9), (90, 90, 65)):
        lens = rng.integers(0, min(top, n) + 1, size=m)
        lens[m // 2] = min(top, n)
        _check(ctx, _csr(lens, n, p, m + b), b, p, [4])


@pytest.mark.parametrize("apps", [[1, 4], [5, 1, 7], [3, 40], [520]])
def test_run_lengths(ctx, apps):
    """Short runs (pass kernels) before and after resident ones, odd counts (the block buffers
    swap roles), and more applications than one launch takes."""
    _check(ctx, synth.incidence_fast(300, 250, 3, 10, 3, P, 5), 8, P, apps)


def test_more_row_batches_than_sms(ctx):
    _check(ctx, synth.incidence_fast(9001, 7003, 3, 10, 10, P, 6), 16, P, [6])


def test_side_by_side(ctx):
    """Handles on several contexts stepped from several threads, while a batch runs on the
    same device: every sequence is the oracle's."""
    mats = [synth.incidence_fast(400 + 100 * i, 300 + 90 * i, 3, 10, 2, P, 20 + i) for i in range(4)]
    errors = []

    def work(mat, seed):
        try:
            c = rr.Context(0)
            _check(c, mat, 8, P, [16, 16, 32], seed)
            c.close()
        except BaseException as e:  # noqa: BLE001 (re-raised below)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(mat, 40 + i)) for i, mat in enumerate(mats)]
    for t in threads:
        t.start()
    pre = [synth.preconditioners(m, n, P, 60 + i) for i, (_, _, _, m, n) in enumerate(mats)]
    vs = [synth.random_vectors(8, mat[4], P, 80 + i) for i, mat in enumerate(mats)]
    bt = rr.Batch(mats, 8, P, [x[0] for x in pre], [x[1] for x in pre], vs, ctx)
    bt.krylov()
    for t in threads:
        t.join()
    assert not errors, errors
    for i, (rowptr, col, val, m, n) in enumerate(mats):
        ref, L, _ = oracle.krylov(rowptr, col, val, m, n, P, pre[i][0], pre[i][1], vs[i], 0,
                                  rr.default_max_nlen(m, n, 8))
        assert np.array_equal(bt.sequence(i), ref[:, :L])
    bt.close()
