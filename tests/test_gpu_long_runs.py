"""Long sequences of a matrix of some hundred thousand columns, width against width: the terms of
the first vectors of a block are those of these vectors alone, so the tcgen05 Gram pass (widths 16
and 32), whose ring of raw tiles goes round thousands of times, is compared with the Gram sums that
the even pass forms on the way (width 8)."""
import numpy as np
import pytest

import rust_rank_b200 as rr
from rust_rank_b200 import synth

pytestmark = pytest.mark.gpu

P = 2013265921


def _pairs(b, upto):
    """Positions of the pairs (i, j), i <= j < upto, in a sequence of width b."""
    return [i * b - i * (i - 1) // 2 + j - i for i in range(upto) for j in range(i, upto)]


@pytest.fixture(scope="module")
def problem(ctx):
    rowptr, col, val, m, n = synth.incidence_fast(600_000, 408_000, 3, 10, 100, P, 3)
    dr, dc = synth.preconditioners(m, n, P, 4)
    dm = rr.CsrMatrix.from_arrays(rowptr, col, val, m, n).to_device(P, ctx)
    yield dm, dr, dc, synth.random_vectors(32, n, P, 5)
    dm.close()


def _terms(problem, b, apps):
    dm, dr, dc, V = problem
    ks = rr.KrylovStream(dm, V[:b], dr, dc, 0)
    seq = np.zeros((b * (b + 1) // 2, 2 * apps + 1), np.uint32)
    ks.step_device(apps)
    ks.fetch(0, 2 * apps + 1, seq)
    block = ks.get_curv()
    ks.close()
    return seq, block


@pytest.mark.parametrize("b,apps", [(16, 24576), (32, 6144)])
def test_width_against_width(problem, b, apps):
    wide, wblock = _terms(problem, b, apps)
    narrow, nblock = _terms(problem, 8, apps)
    assert np.array_equal(wblock[:8], nblock)
    assert np.array_equal(wide[_pairs(b, 8)], narrow)
    again, _ = _terms(problem, b, apps)  # the pairs that width 8 does not have
    assert np.array_equal(wide, again)
