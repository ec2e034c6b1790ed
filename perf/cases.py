"""Performance cases of the block-Wiedemann rank engine.

Each case is one use of the package's public entry points on seeded synthetic
data, from a single application of the operator on a small matrix to the
generator of a long sequence.  ``listed`` gives the fixed cases, ``draw`` one
more of the same ranges, ``prepare`` what a program holds before the call (host
arrays, resident matrices, services), ``run`` one pass, ``work`` the bytes and
operations a pass cannot do without.

Kinds:

* ``next``      -- KrylovStream.next(): one application, the block back on the host
* ``sequence``  -- Krylov sequence of a matrix already on the device, from new
                   preconditioners and a new starting block, terms to the host
* ``end_to_end``-- the same from a host CSR matrix (upload and device build included)
* ``generator`` -- PM_Basis of a sequence on the host
* ``rank``      -- the whole pipeline: host CSR -> sequence -> generator -> rank
* ``batch``     -- many matrices of uneven sizes ranked together
* ``served``    -- requests to a running rank service, all waited for
"""
import math

import numpy as np
import torch

import rust_rank_b200 as rr
from rust_rank_b200 import synth

P = 2013265921   # 15 * 2^27 + 1: products by number-theoretic transform modulo p itself
P_CRT = 27644437  # no long transform: exact integer products joined by CRT
P_MAX = 2147483647  # 2^31 - 1, the largest prime taken; also without a transform


def listed():
    return [
        # one application, the reference's VectorStream::next: latency alone
        {"name": "next_5k_b3", "kind": "next", "matrix": "incidence", "m": 5003, "n": 4001, "b": 3, "p": P},
        # a small rank by itself, at a prime of the reference (CRT products), narrow block
        {"name": "rank_1500_b4_crt", "kind": "rank", "matrix": "incidence", "m": 1501, "n": 1203, "b": 4, "p": P_CRT},
        # the plain single-matrix workload: 20,000^2, 6 entries per row, 500 dependent rows
        {"name": "rank_20k_b8", "kind": "rank", "matrix": "plain", "m": 20000, "n": 20000, "b": 8, "p": P},
        # mid-sized sequence at a ragged width
        {"name": "seq_30k_b5", "kind": "sequence", "matrix": "incidence", "m": 30011, "n": 23017, "b": 5, "p": P_MAX,
         "terms": 4096},
        # the largest matrix of the graph-complex batch (3 to 10 entries per row, no heavy columns)
        {"name": "seq_194k_b16", "kind": "sequence", "matrix": "incidence", "m": 194003, "n": 151007, "b": 16, "p": P,
         "terms": 2048},
        # the large single-matrix workload: 2M x 1.5M, 12 Zipf(1.1) columns per row
        {"name": "seq_zipf_2m_b16", "kind": "sequence", "matrix": "zipf", "m": 2000000, "n": 1500000, "k": 12,
         "s": 1.1, "b": 16, "p": P, "terms": 2048},
        # the same family at half the size and the widest block
        {"name": "seq_zipf_1m_b32", "kind": "sequence", "matrix": "zipf", "m": 1000003, "n": 750007, "k": 12,
         "s": 1.1, "b": 32, "p": P, "terms": 1024},
        # the large matrix from the host: upload, device build and the first terms
        {"name": "e2e_zipf_2m_b16", "kind": "end_to_end", "matrix": "zipf", "m": 2000000, "n": 1500000, "k": 12,
         "s": 1.1, "b": 16, "p": P, "terms": 128},
        # generator of a long sequence
        {"name": "gen_64k_b16", "kind": "generator", "b": 16, "d": 65536, "p": P},
        # generator at the widest block (leaves on the CUDA cores)
        {"name": "gen_1k_b32", "kind": "generator", "b": 32, "d": 1024, "p": P},
        # many small matrices together
        {"name": "batch_24_b8", "kind": "batch", "count": 24, "rmin": 1000, "rmax": 8000, "b": 8, "p": P},
        # requests to a running service
        {"name": "served_6_b8", "kind": "served", "count": 6, "rmin": 4000, "rmax": 16000, "b": 8, "p": P},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case.  Sizes are log-uniform; the sequence length is cut so that
    no drawn case costs more than the longest listed one."""
    kind = rng.choice(["next", "sequence", "sequence", "sequence", "sequence", "end_to_end", "generator", "generator",
                       "rank", "rank", "batch", "served"])
    p = rng.choice([P, P, P, P_CRT, P_MAX])
    if kind == "generator":
        b = rng.choice([1, 2, 4, 5, 8, 12, 16, 16, 24, 32])
        top = 32768 if b <= 8 else 16384 if b <= 16 else 1024
        return {"kind": kind, "b": b, "d": _log_int(rng, 64, top), "p": p}
    if kind == "batch":
        rmax = _log_int(rng, 2000, 8000)
        return {"kind": kind, "count": rng.randint(4, 24), "rmin": rmax // rng.randint(2, 8), "rmax": rmax,
                "b": rng.choice([4, 8, 16]), "p": p}
    if kind == "served":
        rmax = _log_int(rng, 4000, 16000)
        return {"kind": kind, "count": rng.randint(2, 6), "rmin": rmax // rng.randint(2, 4), "rmax": rmax,
                "b": rng.choice([8, 16]), "p": p}
    if kind == "rank":
        m = _log_int(rng, 700, 20000)
        if rng.random() < 0.5:
            return {"kind": kind, "matrix": "plain", "m": m, "n": m, "b": rng.choice([8, 16]), "p": p}
        return {"kind": kind, "matrix": "incidence", "m": m, "n": max(8, int(m * rng.uniform(0.6, 1.0))),
                "b": rng.choice([4, 5, 8, 16]), "p": p}
    b = rng.choice([1, 2, 3, 4, 5, 8, 11, 16, 16, 16, 27, 32])
    if kind == "next" or rng.random() < 0.5:
        m = _log_int(rng, 2000, 200000)
        case = {"kind": kind, "matrix": "incidence", "m": m, "n": max(8, int(m * rng.uniform(0.6, 1.0))), "b": b,
                "p": p}
        nnz = 6.5 * m
    else:
        m, k = _log_int(rng, 50000, 2000000), rng.randint(6, 12)
        case = {"kind": kind, "matrix": "zipf", "m": m, "n": max(64, int(m * rng.uniform(0.5, 1.0))), "k": k,
                "s": round(rng.uniform(0.8, 1.2), 2), "b": b, "p": p}
        nnz = k * m
    if kind == "sequence":
        top = min(4096.0, 8e11 / (nnz * b))
        case["terms"] = 2 * (_log_int(rng, min(256.0, top), top) // 2)
    elif kind == "end_to_end":
        case["terms"] = 2 * rng.randint(8, 64)
    return case


# ---------------------------------------------------------------- inputs
def _zipf(m, n, k, s, p, seed):
    """The matrix of synth.zipf_large (k distinct Zipf(s) columns per row over a
    random column order, values uniform in [1, p), 0.5 % duplicated rows), drawn
    on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    cdf = np.cumsum(np.arange(1, n + 1, dtype=np.float64) ** (-s))
    cdf = torch.from_numpy(cdf / cdf[-1]).cuda()
    colmap = torch.randperm(n, generator=g, device="cuda")

    def fresh(shape):
        u = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)
        return colmap[torch.searchsorted(cdf, u, right=True).clamp_(max=n - 1)]

    dup = m // 200
    base = m - dup
    cols = torch.sort(fresh((base, k)), dim=1).values
    bad = torch.arange(base, device="cuda")
    while True:
        sub = cols[bad]
        rep = torch.zeros_like(sub, dtype=torch.bool)
        rep[:, 1:] = sub[:, 1:] == sub[:, :-1]
        again = rep.any(dim=1)
        bad, sub, rep = bad[again], sub[again], rep[again]
        if bad.numel() == 0:
            break
        cols[bad] = torch.sort(torch.where(rep, fresh(sub.shape), sub), dim=1).values
    vals = torch.randint(1, p, (base, k), generator=g, device="cuda")
    src = torch.randint(0, base, (dup,), generator=g, device="cuda")
    perm = torch.randperm(m, generator=g, device="cuda")
    cols = torch.cat([cols, cols[src]])[perm].to(torch.int32).cpu().numpy().reshape(-1)
    vals = torch.cat([vals, vals[src]])[perm].to(torch.int32).cpu().numpy().view(np.uint32).reshape(-1)
    return np.arange(0, (m + 1) * k, k, dtype=np.int64), cols, vals, m, n


def _matrix(case, seed):
    m, n, p = case["m"], case["n"], case["p"]
    if case["matrix"] == "zipf":
        return _zipf(m, n, case["k"], case["s"], p, seed)
    if case["matrix"] == "plain":
        return synth.plain_single(n=m, k=6, dep_rows=m // 40, p=p, seed=seed)
    return synth.incidence_fast(m, n, 3, 10, n // 100 + 1, p, seed)


def _vectors(m, n, b, p, seed):
    dr, dc = synth.preconditioners(m, n, p, seed + 1)
    return dr, dc, synth.random_vectors(b, n, p, seed + 2)


def _shapes(case):
    """Rows log-uniform in [rmin, rmax], columns 0.6 to 1 of them: a function of the case alone."""
    rng = np.random.default_rng([case["count"], case["rmin"], case["rmax"]])
    rows = np.exp(rng.uniform(math.log(case["rmin"]), math.log(case["rmax"]), case["count"]))
    return [(int(m), max(8, int(m * f))) for m, f in zip(rows, rng.uniform(0.6, 1.0, case["count"]))]


def _many(case, seed):
    mats, drs, dcs, vs = [], [], [], []
    for i, (m, n) in enumerate(_shapes(case)):
        mats.append(synth.incidence_fast(m, n, 3, 10, n // 100 + 1 if i % 8 == 0 else 0, case["p"], seed * 64 + i))
        dr, dc, v = _vectors(m, n, case["b"], case["p"], seed * 64 + i)
        drs.append(dr)
        dcs.append(dc)
        vs.append(v)
    return mats, drs, dcs, vs


def prepare(case, seed):
    kind, p = case["kind"], case["p"]
    st = {"case": case}
    if kind == "generator":
        # a sequence of random symmetric blocks: the generic one (every leaf has full rank)
        b, terms = case["b"], (1 << max(0, (case["d"] - 1).bit_length())) + 1
        st["seq"] = synth.random_vectors(b * (b + 1) // 2, terms, p, seed)
        return st
    if kind in ("batch", "served"):
        st["many"] = _many(case, seed)
        if kind == "served":
            st["server"] = rr.Server(case["b"], p)
        return st
    rowptr, col, val, m, n = _matrix(case, seed)
    st["dr"], st["dc"], st["v"] = _vectors(m, n, case["b"], p, seed)
    csr = rr.CsrMatrix.from_arrays(rowptr, col, val, m, n)
    if kind in ("next", "sequence"):
        st["dm"] = csr.to_device(p)
    else:
        st["csr"] = csr
    if kind == "next":
        st["ks"] = rr.KrylovStream(st["dm"], st["v"], st["dr"], st["dc"], 0)
    return st


# ---------------------------------------------------------------- one pass
def _sequence(st, dm, max_nlen):
    b, p = st["case"]["b"], st["case"]["p"]
    ks = rr.KrylovStream(dm, st["v"], st["dr"], st["dc"], 0)
    seq = np.zeros((b * (b + 1) // 2, max_nlen + 1), np.uint32)
    curv = np.empty_like(st["v"])
    length = rr.main_loop_s_mt2(ks, st["dr"], st["dc"], curv, st["v"], seq, 0, max_nlen, theprime=p)
    ks.close()
    return seq[:, :length], curv


def run(st):
    case = st["case"]
    kind, p = case["kind"], case["p"]
    if kind == "next":
        return [w.view(np.int32) for w in st["ks"].next()]
    if kind == "sequence":
        return [x.view(np.int32) for x in _sequence(st, st["dm"], case["terms"])]
    if kind == "generator":
        M, delta = rr.PM_Basis(st["seq"], case["d"], p)
        return [M.view(np.int32), delta]
    if kind == "batch":
        mats, drs, dcs, vs = st["many"]
        bt = rr.Batch(mats, case["b"], p, drs, dcs, vs)
        ranks = bt.ranks()
        seqs = [bt.sequence(i).view(np.int32) for i in range(len(mats))]
        bt.close()
        return [ranks, *seqs]
    if kind == "served":
        ids = [st["server"].submit(*mat, dr, dc, v) for mat, dr, dc, v in zip(*st["many"])]
        return np.array([st["server"].result(i)[0] for i in ids])
    dm = st["csr"].to_device(p)
    if kind == "end_to_end":
        out = _sequence(st, dm, case["terms"])
        dm.close()
        return [x.view(np.int32) for x in out]
    seq, _ = _sequence(st, dm, rr.default_max_nlen(case["m"], case["n"], case["b"]))
    dm.close()
    d = 1
    while 2 * d <= seq.shape[1] - 1:
        d *= 2
    M, delta = rr.PM_Basis(seq, d, p)
    return [seq.view(np.int32), M.view(np.int32), delta, rr.analyze_pm_basis(M, delta, p)]


def exact(case, seed):
    """Every output is a residue, a degree or a rank: whole numbers, equal or wrong."""
    return None


# ---------------------------------------------------------------- what a pass cannot do without
def _krylov_work(m, n, nnz, b, apps):
    # CSR of A and A^T read once, both dense blocks read and written once;
    # one modular multiply-add = 2 operations
    by = 16.0 * nnz + 4.0 * (m + n + 2) + 8.0 * b * (m + n)
    return apps * by, apps * (4.0 * nnz * b + (m + n) * b * (b + 1.0))


def _generator_work(b, d):
    # sequence in, basis out; per order the elimination of a 2b x b block beside
    # its 2b transform columns, and log2(d) levels of matrix products
    dd = 1 << max(0, (d - 1).bit_length())
    m = 2 * b
    levels = max(1, dd.bit_length() - 1)
    flops = dd * 2.0 * (m * b * 1.5 * m) + dd * levels * (2.0 * m * m * m + 2.0 * m * m * b + 10.0 * m * m * levels)
    return 4.0 * (b * (b + 1) / 2 * dd + m * m * (dd + 1)), flops


def work(case):
    kind, b = case["kind"], case["b"]
    if kind == "generator":
        by, fl = _generator_work(b, case["d"])
        return {"bytes": by, "flops": fl}

    def terms_of(m, n):
        return rr.default_max_nlen(m, n, b)

    def whole(m, n, nnz):
        t = terms_of(m, n)
        kb, kf = _krylov_work(m, n, nnz, b, t / 2)
        gb, gf = _generator_work(b, max(1, t // 2))
        return 12.0 * nnz + kb + gb, kf + gf

    if kind in ("batch", "served"):
        by = fl = 0.0
        for m, n in _shapes(case):
            x, y = whole(m, n, 6.5 * m)
            by, fl = by + x, fl + y
        return {"bytes": by, "flops": fl}
    m, n = case["m"], case["n"]
    nnz = {"zipf": case.get("k", 0), "plain": 6.3, "incidence": 6.5}[case["matrix"]] * m
    if kind == "rank":
        by, fl = whole(m, n, nnz)
    elif kind == "next":
        by, fl = _krylov_work(m, n, nnz, b, 1)
        by += 4.0 * b * n
    else:
        by, fl = _krylov_work(m, n, nnz, b, case["terms"] / 2)
        by += 8.0 * b * n + 4.0 * (m + n)
        if kind == "end_to_end":
            by += 12.0 * nnz + 16.0 * nnz
    return {"bytes": by, "flops": fl}
