"""Resident runs of several contexts side by side (resident.cu): every sequence is the oracle's
whatever shares of the device the runs get, and the contexts do not queue up behind one another."""
import threading
import time

import numpy as np
import pytest

import oracle
import rust_rank_b200 as rr
from rust_rank_b200 import synth

pytestmark = pytest.mark.gpu

P = 2013265921


class Stepper:
    def __init__(self, m, b, seed):
        self.mat = synth.incidence_fast(m, int(0.8 * m), 3, 10, 2, P, seed)
        m, n = self.mat[3], self.mat[4]
        self.dr, self.dc = synth.preconditioners(m, n, P, seed + 1)
        self.V = synth.random_vectors(b, n, P, seed + 2)
        self.ctx = rr.Context(0)
        self.dm = rr.CsrMatrix.from_arrays(*self.mat).to_device(P, self.ctx)
        self.ks = rr.KrylovStream(self.dm, self.V, self.dr, self.dc, 0)

    def run(self, pieces):
        for k in pieces:
            self.ks.step_device(k)
        self.ctx.synchronize()

    def check(self, apps):
        b = self.V.shape[0]
        seq = np.zeros((b * (b + 1) // 2, 2 * apps + 1), np.uint32)
        self.ks.fetch(0, 2 * apps + 1, seq)
        ref, _, cv = oracle.krylov(*self.mat, P, self.dr, self.dc, self.V, 0, 2 * apps)
        assert np.array_equal(seq, ref) and np.array_equal(self.ks.get_curv(), cv)

    def close(self):
        self.ks.close()
        self.dm.close()
        self.ctx.close()


def _together(steppers, pieces):
    """Seconds for all of them to run their pieces, a thread each."""
    gate = threading.Barrier(len(steppers) + 1)

    def work(s):
        gate.wait()
        s.run(pieces)

    threads = [threading.Thread(target=work, args=(s,)) for s in steppers]
    for t in threads:
        t.start()
    gate.wait()
    t0 = time.perf_counter()
    for t in threads:
        t.join()
    return time.perf_counter() - t0


@pytest.mark.parametrize("shapes", [[(60, 3)] * 20, [(2500, 4), (900, 8), (3000, 16), (40, 1), (5000, 16), (700, 7)],
                                    [(12000, 16), (300, 4), (9000, 8), (11000, 12)]])
def test_runs_of_mixed_sizes(shapes):
    """More contexts than shares, and shares of different sizes in changing company."""
    steppers = [Stepper(m, b, 10 * i) for i, (m, b) in enumerate(shapes)]
    pieces = [4, 9, 1, 16, 5, 3, 12]
    _together(steppers, pieces)
    for s in steppers:
        s.check(sum(pieces))
        s.close()


def test_contexts_run_side_by_side():
    """Eight contexts together take well below eight times one of them (2 times measured; one after
    the other, 7.6 times)."""
    steppers = [Stepper(700, 4, 10 * i) for i in range(8)]
    pieces = [128] * 8
    one = min(_together(steppers[:1], pieces) for _ in range(8))
    eight = min(_together(steppers, pieces) for _ in range(8))
    for s in steppers:
        s.close()
    assert eight < 5 * one, (one, eight)
