"""Device-side waits that run out: the kernel ends by itself, the calls that read its results
report the time-out, and the context goes on working.  The waits are made to run out by
expecting more arrivals than come, with a short limit; nothing faults or hangs."""
import contextlib
import time

import numpy as np
import pytest

import oracle
import rust_rank_b200 as rr
from rust_rank_b200 import synth

pytestmark = pytest.mark.gpu

P = 2013265921
ETIMEOUT = 5


@pytest.fixture(scope="module")
def module_ctx():
    return rr.Context(0)


@pytest.fixture
def own_ctx(module_ctx):
    yield module_ctx
    module_ctx.set_waits()


def _problem(m, b, seed=3):
    rowptr, col, val, m, n = synth.incidence_fast(m, int(0.8 * m), 3, 10, 2, P, seed)
    dr, dc = synth.preconditioners(m, n, P, seed + 1)
    return (rowptr, col, val, m, n), dr, dc, synth.random_vectors(b, n, P, seed + 2)


@contextlib.contextmanager
def _stream(ctx, prob):
    mat, dr, dc, V = prob
    dm = rr.CsrMatrix.from_arrays(*mat).to_device(P, ctx)
    ks = rr.KrylovStream(dm, V, dr, dc, 0)
    yield ks
    ks.close()
    dm.close()


@contextlib.contextmanager
def rr_server(b):
    srv = rr.Server(b, P, lanes=2, workers=2)
    yield srv
    srv.close()


def _timed_out(call, *args):
    try:
        call(*args)
    except rr.RRError as e:
        assert e.status == ETIMEOUT
    else:
        pytest.fail("no error")


def _works(ctx, prob):
    """A new handle on the same context computes the oracle's sequence."""
    mat, dr, dc, V = prob
    b = V.shape[0]
    seq = np.zeros((b * (b + 1) // 2, 17), np.uint32)
    with _stream(ctx, prob) as ks:
        ks.step_device(8)
        ks.fetch(0, 17, seq)
        ref, _, cv = oracle.krylov(*mat, P, dr, dc, V, 0, 16)
        assert np.array_equal(seq, ref[:, :17])
        assert np.array_equal(ks.get_curv(), cv)


@pytest.mark.parametrize("m,b", [(12, 1), (700, 4), (700, 8), (700, 16), (20000, 8), (20000, 16)])
def test_grid_barrier_of_a_resident_run(own_ctx, m, b):
    """Every warp of every CTA leaves the run, whatever it was doing when the wait ran out."""
    prob = _problem(m, b)
    seq = np.zeros((b * (b + 1) // 2, 32), np.uint32)
    with _stream(own_ctx, prob) as ks:
        own_ctx.set_waits(0.02, 1)
        t0 = time.perf_counter()
        for apps in (4, 9, 30):
            ks.step_device(apps)
        own_ctx.synchronize()
        assert time.perf_counter() - t0 < 1.5
        _timed_out(ks.fetch, 0, 9, seq)
        own_ctx.set_waits()
        ks.step_device(5)
        _timed_out(ks.fetch, 0, 9, seq)  # the handle's state is lost
    _works(own_ctx, prob)


@pytest.mark.parametrize("m,b", [(700, 8), (700, 16), (90000, 16)])
def test_block_of_a_run_that_gave_up(own_ctx, m, b):
    """A block that a given-up run left half advanced is not returned as valid: neither by get_curv nor
    by next(), which at width 16 is a resident run of its own for small matrices."""
    prob = _problem(m, b)
    with _stream(own_ctx, prob) as ks:
        own_ctx.set_waits(0.02, 1)
        ks.step_device(4)
        _timed_out(ks.get_curv)
        own_ctx.set_waits()
        _timed_out(ks.get_curv)
        _timed_out(ks.next)
    if b == 16 and m == 700:
        with _stream(own_ctx, prob) as ks:
            own_ctx.set_waits(0.02, 1)
            _timed_out(ks.next)
            own_ctx.set_waits()
    _works(own_ctx, prob)


@pytest.mark.parametrize("terms", [9, 1023, 1024, 5001])
def test_terms_of_a_run_that_gave_up(own_ctx, terms):
    """The caller's array keeps what it held, whatever the length of the fetch."""
    b = 8
    prob = _problem(700, b)
    with _stream(own_ctx, prob) as ks:
        ks.step_device(4)
        seq = np.full((b * (b + 1) // 2, terms + 2), 7, np.uint32)
        ks.fetch(0, 9, seq)
        head = seq[:, :9].copy()
        own_ctx.set_waits(0.02, 1)
        ks.step_device(terms // 2)
        _timed_out(ks.fetch, 0, terms, seq)
        own_ctx.set_waits()
        assert np.array_equal(seq[:, :9], head) and (seq[:, 9:] == 7).all()


@pytest.mark.parametrize("b", [8, 16])
def test_served_request_whose_run_gave_up(b):
    """The request fails instead of returning a rank of terms that were never computed; the one solved
    together with it, and later ones of the same lane, return theirs."""
    (rowptr, col, val, m, n), dr, dc, V = _problem(700, b)
    with rr_server(b) as srv:
        want = rr.block_wiedemann_rank(rr.CsrMatrix.from_arrays(rowptr, col, val, m, n), b, P, dr, dc, V)
        srv.set_waits(0, 0.02, 1)
        ids = [srv.submit(rowptr, col, val, m, n, dr, dc, V) for _ in range(2)]  # one per lane
        with pytest.raises(rr.RRError, match="gave up") as e:
            srv.result(ids[0])
        assert e.value.status != ETIMEOUT  # which would say that it is not finished
        assert srv.result(ids[1])[0] == want
        srv.set_waits(0)
        ids = [srv.submit(rowptr, col, val, m, n, dr, dc, V) for _ in range(4)]
        assert [srv.result(i)[0] for i in ids] == [want] * 4
        assert srv.stats()["completed"] == 6


@pytest.mark.parametrize("b,d", [(1, 1), (2, 2), (4, 64), (8, 256), (16, 4), (16, 256), (32, 16), (32, 128)])
def test_hand_offs_of_leaf_blocks(own_ctx, b, d):
    """Every CTA of the cluster ends, the blocks after the first do not wait as long again, and the context's
    next generator is the oracle's."""
    rng = np.random.default_rng(b + d)
    seqs = [rng.integers(0, P, size=(b * (b + 1) // 2, d + 1)).astype(np.uint32) for _ in range(2)]
    own_ctx.set_waits(0.3, 1)
    t0 = time.perf_counter()
    _timed_out(rr.PM_Basis_batch, seqs, d, P, own_ctx)
    assert time.perf_counter() - t0 < 1.5  # up to eight blocks
    own_ctx.set_waits()
    M, delta = rr.PM_Basis(seqs[0], d, P, own_ctx)
    Mo, do = oracle.pm_basis(seqs[0], b, d, P)
    assert np.array_equal(M, Mo.astype(np.uint32)) and np.array_equal(delta, do)


def test_arguments(own_ctx):
    for limit, missing in ((0.0, 0), (11.0, 0), (float("nan"), 0), (1.0, -1)):
        with pytest.raises(rr.RRError):
            own_ctx.set_waits(limit, missing)
