"""Blocks into arrays whose pages are there already and into ones that are not, around the sizes
where the copy changes its way (upload.cpp: 4 MB, and 8 MB for touched pages), at any alignment."""
import mmap

import numpy as np
import pytest

import rust_rank_b200 as rr
from rust_rank_b200 import synth

pytestmark = pytest.mark.gpu

P = 2013265921


@pytest.mark.parametrize("mb", [4.0, 4.2, 7.9, 8.4])
def test_pages_there_and_not(ctx, mb):
    b = 8
    n = int(mb * (1 << 20) / 4 / b) + 3
    V = synth.random_vectors(b, n, P, 1)
    dr, dc = synth.preconditioners(1, n, P, 2)
    dm = rr.CsrMatrix.from_arrays(np.array([0, 1], np.int64), [0], [1], 1, n).to_device(P, ctx)
    ks = rr.KrylovStream(dm, V, dr, dc, 0)
    nbytes = 4 * b * n
    for touched in (0.0, 0.3, 0.7, 1.0):
        for offset in (0, 4, 4092):
            raw = np.frombuffer(mmap.mmap(-1, nbytes + 8192), np.uint8)
            raw[: int(touched * raw.size)] = 7
            out = raw[offset : offset + nbytes].view(np.uint32).reshape(b, n)
            ks.get_curv(out)
            assert np.array_equal(out, V)
            assert (raw[:offset] == (7 if touched else 0)).all()
            assert (raw[offset + nbytes :] == (7 if touched == 1.0 else 0)).all()
    ks.close()
    dm.close()
