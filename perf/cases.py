"""Timed cases of the search path, through its public entry points.

Three kinds of call are covered, over the sizes the benchmark configurations
and the tests use:

  search   one search::run: over a resident database and batch, as a batch of
           tagged requests (the server's call), or from host buffers
  blastx   reads translated on the device, searched and merged per read
  stages   the per-stage entry points from host buffers: seed_build,
           seed_join, xdrop, extend_scores, extend_span

Sequences follow the benchmark generator: lognormal lengths, residues from the
BLOSUM62 background, 2 % of the database sequences with a homopolymer run, and
mutated query segments (25-70 % identity, 2 % indels) planted in database
sequences.  Everything is drawn from the seed; the draws are whole-array numpy
calls, so that preparing a case is quick.
"""
import ctypes as C
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "diamond-rust_b200"))

import drgpu  # noqa: E402
from drgpu import serve, synth  # noqa: E402

# Reference DP cells per (query letter x database letter), measured per preset
# on the generator below; the path's unavoidable arithmetic is estimated from
# them.
CELLS_PER_PAIR = {"fast": 3.9e-5, "default": 3.2e-4, "mid-sensitive": 4.7e-3, "sensitive": 4.8e-2,
                  "more-sensitive": 4.8e-2, "very-sensitive": 0.14, "ultra-sensitive": 0.40}
OPS_PER_CELL = 8  # diagonal add, two gap adds and maxima each for E and F, three maxima for H
HSP_BYTES = C.sizeof(drgpu.Hsp)
HSP_FIELDS = ("query", "subject", "frame", "score", "q_begin", "q_end", "s_begin", "s_end", "bits", "evalue",
              "identities", "positives", "mismatches", "gap_openings", "gaps", "length", "ops_offset", "n_ops")


def listed():
    return [
        # one query against a small proteome: the latency of a search, its launches and waits
        {"name": "one_query_default", "kind": "search", "via": "resident", "queries": 1, "q_mean": 497, "db": 7860,
         "db_mean": 288, "preset": "default", "chunks": -1, "index": False, "matrix": "BLOSUM62", "max_hsps": 1,
         "evalue": 1e-3},
        # a server's merged batch: several small requests on a database whose seed index is resident
        {"name": "requests_sensitive_indexed", "kind": "search", "via": "requests", "queries": 61, "q_mean": 350,
         "db": 7860, "db_mean": 288, "requests": 7, "preset": "sensitive", "chunks": -1, "index": True,
         "matrix": "BLOSUM62", "max_hsps": 1, "evalue": 1e-3},
        # the flagship batch
        {"name": "batch_sensitive", "kind": "search", "via": "resident", "queries": 1000, "q_mean": 350, "db": 7860,
         "db_mean": 288, "preset": "sensitive", "chunks": 1, "index": False, "matrix": "BLOSUM62", "max_hsps": 1,
         "evalue": 1e-3},
        # the other named preset of that batch, an odd count of queries
        {"name": "batch_very_sensitive", "kind": "search", "via": "resident", "queries": 501, "q_mean": 350,
         "db": 7860, "db_mean": 288, "preset": "very-sensitive", "chunks": 1, "index": False, "matrix": "BLOSUM62",
         "max_hsps": 1, "evalue": 1e-3},
        # a few long proteins (up to 3,000 aa) at the deepest preset, another matrix, several HSPs per pair: the
        # drop-in call from host buffers
        {"name": "host_ultra_long", "kind": "search", "via": "host", "queries": 13, "q_mean": 900, "db": 1001,
         "db_mean": 500, "preset": "ultra-sensitive", "chunks": -1, "index": False, "matrix": "BLOSUM80",
         "max_hsps": 5, "evalue": 10.0},
        # many queries against a larger database at the default sensitivity, from host buffers
        {"name": "host_many_default", "kind": "search", "via": "host", "queries": 20000, "q_mean": 350, "db": 60000,
         "db_mean": 288, "preset": "default", "chunks": -1, "index": False, "matrix": "BLOSUM62", "max_hsps": 1,
         "evalue": 1e-3},
        # short nucleotide reads against a protein database, the whole call from the reads' bytes
        {"name": "blastx_fast", "kind": "blastx", "reads": 20000, "db": 20000, "preset": "fast"},
        # the stage calls of a program that keeps its own orchestration
        {"name": "seed_build_db", "kind": "seed_build", "seqs": 7860, "mean": 288, "shape": "1011110111",
         "reduction": 0, "cut": 5.545177444479562},
        {"name": "seed_join_batch", "kind": "seed_join", "queries": 1000, "q_mean": 350, "db": 7860,
         "shape": "1101110101101111", "reduction": 0, "cut": 0.0},
        {"name": "xdrop_hits", "kind": "xdrop", "jobs": 400001, "queries": 300, "q_mean": 350, "db": 4000},
        {"name": "extend_scores_bands", "kind": "extend_scores", "jobs": 200003, "queries": 300, "q_mean": 350,
         "db": 4000, "matrix": "BLOSUM62"},
        {"name": "extend_span_hsps", "kind": "extend_span", "jobs": 3001, "queries": 700, "q_mean": 350, "db": 4000,
         "matrix": "BLOSUM62"},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    most = max(work(c)["flops"] for c in listed() if c["kind"] == "search")
    kind = rng.choice(["search", "search", "search", "blastx", "seed_build", "seed_join", "xdrop", "extend_scores",
                       "extend_span"])
    if kind == "search":
        via = rng.choice(["resident", "requests", "host"])
        c = {"kind": kind, "via": via, "queries": _log_int(rng, 1, 4000),
             "q_mean": rng.choice([120, 350, 350, 497, 700]), "db": _log_int(rng, 500, 20000),
             "db_mean": rng.choice([200, 288, 288, 400]),
             "preset": rng.choice(["fast", "default", "mid-sensitive", "sensitive", "more-sensitive",
                                   "very-sensitive", "ultra-sensitive"]),
             "chunks": rng.choice([-1, 1, 3]), "index": via != "host" and rng.random() < 0.5,
             "matrix": rng.choice(["BLOSUM62", "BLOSUM62", "BLOSUM45", "BLOSUM80", "PAM70"]),
             "max_hsps": rng.choice([1, 1, 3]), "evalue": rng.choice([1e-3, 1e-3, 1.0])}
        if via == "requests":
            c["requests"] = 1 + rng.randrange(12)
        while work(c)["flops"] > most and c["queries"] > 1:
            c["queries"] = (c["queries"] + 1) // 2
        return c
    if kind == "blastx":
        return {"kind": kind, "reads": _log_int(rng, 50, 20000), "db": _log_int(rng, 500, 20000),
                "preset": rng.choice(["fast", "default"])}
    if kind == "seed_build":
        # the shapes of the presets, their reductions and complexity cuts
        shape, red, per_letter = rng.choice([("1101110101101111", 0, 0.9), ("111101110111", 0, 0.8),
                                             ("1011110111", 0, 1.0), ("11110111", 1, 1.0), ("1111111", 0, 1.0)])
        return {"kind": kind, "seqs": _log_int(rng, 30, 7860), "mean": rng.choice([120, 288, 350]), "shape": shape,
                "reduction": red, "cut": float(per_letter * np.log(2) * shape.count("1"))}
    if kind == "seed_join":
        return {"kind": kind, "queries": _log_int(rng, 5, 1000), "q_mean": rng.choice([120, 350]),
                "db": _log_int(rng, 100, 7860), "shape": rng.choice(["1101110101101111", "111101110111"]),
                "reduction": 0, "cut": 0.0}
    c = {"kind": kind, "jobs": _log_int(rng, 20, {"xdrop": 400000, "extend_scores": 200000, "extend_span": 3000}[kind]),
         "queries": _log_int(rng, 5, 700), "q_mean": rng.choice([120, 350, 497]), "db": _log_int(rng, 200, 4000)}
    if kind != "xdrop":
        c["matrix"] = rng.choice(["BLOSUM62", "BLOSUM45", "PAM70"])
    return c


# ---- inputs -----------------------------------------------------------------
def _pick_table(p, n):
    """n equally likely slots holding the indices of p in its proportions."""
    edges = np.round(np.cumsum(p) * n).astype(np.int64)
    return np.searchsorted(edges, np.arange(n), side="right").clip(0, len(p) - 1).astype(np.uint8)


_RESIDUES = _pick_table(synth.BACKGROUND, 1 << 16)
_TARGET = synth.BACKGROUND[:, None] * synth.BACKGROUND[None, :] * np.exp(synth.LAMBDA_U * synth.B62)
np.fill_diagonal(_TARGET, 0.0)
_SUBSTITUTE = np.stack([_pick_table(row / row.sum(), 1 << 12) for row in _TARGET])


def _residues(rng, n):
    return _RESIDUES[rng.integers(0, 1 << 16, size=int(n), dtype=np.uint16)]


def _offsets(lengths):
    off = np.zeros(len(lengths) + 1, np.uint64)
    off[1:] = np.cumsum(lengths)
    return off


def _proteins(rng, n, mean, lo, hi, homopolymers=0.0):
    lens = synth.lognormal_lengths(rng, n, mean, lo, hi)
    off = _offsets(lens)
    letters = _residues(rng, int(off[-1]))
    for i in np.nonzero(rng.random(n) < homopolymers)[0]:
        run = min(int(rng.integers(10, 31)), int(lens[i]))
        at = int(off[i]) + int(rng.integers(0, lens[i] - run + 1))
        letters[at:at + run] = rng.integers(0, 20)
    return letters, off


def _within(lens):
    """0 .. lens[i] - 1 for each i, one after the other."""
    ends = np.cumsum(lens)
    return np.arange(int(ends[-1]) if len(ends) else 0) - np.repeat(ends - lens, lens)


def _plant(rng, db, db_off, q, q_off, per_query):
    """Writes mutated query segments over parts of distinct database sequences;
    returns (query, subject, query start, subject start, letters) of each."""
    nq, ndb = len(q_off) - 1, len(db_off) - 1
    n = min(ndb, per_query * nq)
    query = np.arange(n) % nq
    subject = rng.permutation(ndb)[:n]
    qlen = (q_off[query + 1] - q_off[query]).astype(np.int64)
    slen = (db_off[subject + 1] - db_off[subject]).astype(np.int64)
    seg = (np.minimum(30, qlen) + rng.random(n) * (qlen - np.minimum(30, qlen) + 1)).astype(np.int64)
    seg = np.minimum(seg, slen)
    q_start = (rng.random(n) * (qlen - seg + 1)).astype(np.int64)
    s_start = (rng.random(n) * (slen - seg + 1)).astype(np.int64)
    own = np.repeat(np.arange(n), seg)
    src = q[np.repeat(q_off[query].astype(np.int64) + q_start, seg) + _within(seg)]
    keep = rng.random(len(src)) < rng.uniform(0.25, 0.70, n)[own]
    src = np.where(keep, src, _SUBSTITUTE[src, rng.integers(0, 1 << 12, len(src))])
    # indels: 2 % of the sites, geometric lengths of mean 3, half of them deletions
    count = np.ones(len(src), np.int64)
    site = np.nonzero(rng.random(len(src)) < 0.02)[0]
    length = rng.geometric(1 / 3, len(site))
    is_del = rng.random(len(site)) < 0.5
    cover = np.zeros(len(src) + 1, np.int64)
    np.add.at(cover, site[is_del], 1)
    np.add.at(cover, np.minimum(site[is_del] + length[is_del], len(src)), -1)
    count[site[~is_del]] += length[~is_del]
    count[np.cumsum(cover[:-1]) > 0] = 0
    out = np.repeat(src, count)
    inserted = _within(count) > 0
    out[inserted] = _residues(rng, int(inserted.sum()))
    got = np.bincount(own, weights=count, minlength=n).astype(np.int64)
    at = _within(got)
    fits = at < np.repeat(slen - s_start, got)
    db[(np.repeat(db_off[subject].astype(np.int64) + s_start, got) + at)[fits]] = out[fits]
    return query, subject, q_start, s_start, seg


def _workload(case, rng):
    q, q_off = _proteins(rng, case["queries"], case["q_mean"], 20, 3000)
    db, db_off = _proteins(rng, case["db"], case.get("db_mean", 288), 30, 5000, 0.02)
    return q, q_off, db, db_off, _plant(rng, db, db_off, q, q_off, 5)


def _reads(rng, n, db, db_off):
    """Reads of 150-300 nt: 30 % are coding fragments of database sequences on a
    random strand with 1 % substitutions, the rest random."""
    lens = rng.integers(150, 301, n)
    off = _offsets(lens)
    nt = rng.integers(0, 4, int(off[-1]), dtype=np.uint8)
    codons = [[i for i, a in enumerate(synth.CODON_TABLE) if a == synth.AA[r]] for r in range(20)]
    table = np.array([(c * 12)[:12] for c in codons], np.uint8)  # T, C, A, G order
    slen = np.diff(db_off.astype(np.int64))
    for i in np.nonzero(rng.random(n) < 0.30)[0]:
        s = int(rng.integers(0, len(slen)))
        n_aa = int(min(lens[i] // 3, slen[s]))
        a = int(db_off[s]) + int(rng.integers(0, slen[s] - n_aa + 1))
        cod = table[db[a:a + n_aa], rng.integers(0, 12, n_aa)]
        x = np.stack([cod // 16, cod // 4 % 4, cod % 4], axis=1).reshape(-1)
        if rng.random() < 0.5:
            x = (x ^ 2)[::-1]  # T-A and C-G are two apart
        nt[int(off[i]):int(off[i]) + 3 * n_aa] = x
    subs = rng.random(len(nt)) < 0.01
    nt[subs] = rng.integers(0, 4, int(subs.sum()))
    return np.frombuffer(b"TCAG", np.uint8)[nt], off


def _jobs(case, rng, homologs, q_off, db_off):
    """(query, subject, query position, subject position): one in five on a
    planted homolog's diagonal, the others anywhere."""
    n = case["jobs"]
    hq, hs, hq0, hs0, seg = homologs
    query = rng.integers(0, len(q_off) - 1, n)
    subject = rng.integers(0, len(db_off) - 1, n)
    qlen = np.diff(q_off.astype(np.int64))
    slen = np.diff(db_off.astype(np.int64))
    pick = rng.integers(0, len(hq), n)
    true = rng.random(n) < 0.2
    query = np.where(true, hq[pick], query)
    subject = np.where(true, hs[pick], subject)
    u = rng.random(n)
    qa = np.where(true, hq0[pick] + (u * seg[pick]).astype(np.int64), (u * qlen[query]).astype(np.int64))
    sa = np.where(true, hs0[pick] + (u * seg[pick]).astype(np.int64), (rng.random(n) * slen[subject]).astype(np.int64))
    return query, subject, qa, sa, qlen[query]


def _span_jobs(case, rng, homologs, q_off, db_off):
    query, subject, qa, sa, qlen = _jobs(case, rng, homologs, q_off, db_off)
    # gapped.rs:27-32 half-widths; one band in ten is a merge of several diagonals
    half = np.array([12, 16, 30, 30, 30, 40, 64, 64])[np.searchsorted([50, 100, 150, 200, 250, 350, 500], qlen,
                                                                      side="right")]
    extra = np.where(rng.random(len(qa)) < 0.1, rng.integers(0, 4 * half + 1), 0)
    jobs = np.zeros(len(qa), np.dtype(drgpu.SpanJob))
    jobs["query"], jobs["subject"] = query, subject
    jobs["d0"], jobs["d1"] = qa - sa - half, qa - sa + half + extra
    # bands of a query follow one another, as a program that walks its queries lists them
    return jobs[np.argsort(query, kind="stable")]


_CTX = None


def _ctx():
    """The program's one device context."""
    global _CTX
    if _CTX is None:
        _CTX = drgpu.Context(0)
    return _CTX


class _State:
    """The inputs and handles of a case, and host buffers that take its results (a
    caller's arena: results that are fewer leave the rest as it was, zero)."""
    db = batch = None

    def __init__(self, case):
        self.case = case

    def records(self, name, n, dtype):
        setattr(self, name, np.zeros(int(n), dtype))

    def hsp_records(self, rows, lists):
        self.records("hsps", rows, np.dtype(drgpu.Hsp))
        self.records("ops", 16 * rows, np.uint32)
        self.records("list_offsets", lists + 1, np.uint64)

    def __del__(self):
        try:
            for x in (self.batch, self.db):
                if x is not None:
                    x.close()
        except Exception:
            pass


def prepare(case, seed):
    rng = np.random.Generator(np.random.PCG64([seed, 20]))
    s = _State(case)
    kind = case["kind"]
    if kind == "search":
        q, q_off, db, db_off, _ = _workload(case, rng)
        n = len(q_off) - 1
        s.hsp_records(64 + 12 * n * case["max_hsps"], n)
        s.cfg = drgpu.make_config(sensitivity=case["preset"], matrix=case["matrix"], evalue=case["evalue"],
                                  max_hsps=case["max_hsps"],
                                  index_chunks=None if case["chunks"] < 0 else case["chunks"])
        if case["via"] == "host":
            s.arrays = (db, db_off, q, q_off, np.arange(n, dtype=np.uint32), np.zeros(n, np.uint8))
            return s
        s.db = drgpu.ResidentDb(_ctx(), db, db_off, index_budget=(8 << 30) if case["index"] else 0)
        if case["via"] == "resident":
            s.batch = drgpu.ResidentBatch(_ctx(), q, q_off)
        else:
            cuts = np.sort(rng.integers(0, n + 1, min(case["requests"], n) - 1))
            seqs = [q[int(q_off[i]):int(q_off[i + 1])] for i in range(n)]
            s.requests = [serve.Request(k, case["preset"], seqs[a:b])
                          for k, (a, b) in enumerate(zip([0, *cuts], [*cuts, n]))]
    elif kind == "blastx":
        db, db_off = _proteins(rng, case["db"], 288, 30, 5000, 0.02)
        s.nt, s.nt_off = _reads(rng, case["reads"], db, db_off)
        s.hsp_records(64 + case["reads"], case["reads"])
        s.records("frame_query", 6 * case["reads"], np.uint32)
        s.records("frame_index", 6 * case["reads"], np.uint8)
        s.cfg = drgpu.make_config(sensitivity=case["preset"])
        s.db = drgpu.ResidentDb(_ctx(), db, db_off)
    elif kind == "seed_build":
        s.letters, s.off = _proteins(rng, case["seqs"], case["mean"], 20, 5000, 0.02)
        s.records("entries", 8000 + 1.5 * case["seqs"] * case["mean"], np.dtype(drgpu.SeedEntry))
    elif kind == "seed_join":
        q, q_off, db, db_off, _ = _workload(case, rng)
        s.q, s.r = (_seed_build(case, x, off, np.zeros(len(x), np.dtype(drgpu.SeedEntry)))
                    for x, off in ((q, q_off), (db, db_off)))
        s.records("hits", 20000 + 40 * case["queries"], np.dtype(drgpu.SeedHit))
    else:
        s.q, s.q_off, s.db_letters, s.db_off, homologs = _workload(case, rng)
        if kind == "extend_span":
            s.records("ops", 64 + 24 * case["jobs"], np.uint32)
        if kind == "xdrop":
            query, subject, qa, sa, _ = _jobs(case, rng, homologs, s.q_off, s.db_off)
            s.jobs = np.zeros(len(qa), np.dtype(drgpu.XdropJob))
            s.jobs["query"], s.jobs["subject"], s.jobs["qa"], s.jobs["sa"] = query, subject, qa, sa
        else:
            s.jobs = _span_jobs(case, rng, homologs, s.q_off, s.db_off)
    return s


# ---- one pass ---------------------------------------------------------------
def _p(a, ctype):
    return a.ctypes.data_as(C.POINTER(ctype))


def _into(buf, ptr, n):
    """The first n records at ptr, which the library allocated, copied into buf."""
    n = min(int(n), len(buf))
    if n:
        C.memmove(buf.ctypes.data, ptr, n * buf.itemsize)
    return n


def _result_columns(s, res):
    _into(s.hsps, res.hsps, res.n_hsps)
    _into(s.ops, res.ops, res.n_ops)
    _into(s.list_offsets, res.target_offsets, res.n_targets + 1)
    return _hsp_columns(s)


def _hsp_columns(s):
    return {**{f: s.hsps[f] for f in HSP_FIELDS}, "target_offsets": s.list_offsets, "ops": s.ops}


def _seed_build(case, letters, off, buf):
    ctx = _ctx()
    out, n = C.POINTER(drgpu.SeedEntry)(), C.c_uint64()
    ctx._check(ctx.lib.drg_seed_build(ctx.h, _p(letters, C.c_uint8), _p(off, C.c_uint64), len(off) - 1,
                                      case["shape"].encode(), case["reduction"], 0, case["cut"], C.byref(out),
                                      C.byref(n)))
    taken = _into(buf, out, n.value)
    ctx.lib.drg_free(out)
    return buf[:taken]


def _searched(s):
    ctx, case = _ctx(), s.case
    res = drgpu.Result()
    try:
        if case["via"] == "host":
            db, db_off, q, q_off, query, frame = s.arrays
            ctx._check(ctx.lib.drg_search_run(ctx.h, _p(db, C.c_uint8), _p(db_off, C.c_uint64), len(db_off) - 1,
                                              _p(q, C.c_uint8), _p(q_off, C.c_uint64), _p(query, C.c_uint32),
                                              _p(frame, C.c_uint8), len(q_off) - 1, C.byref(s.cfg), C.byref(res)))
        else:
            ctx._check(ctx.lib.drg_search_batch(ctx.h, s.db.h, s.batch.h, C.byref(s.cfg), C.byref(res)))
        return _result_columns(s, res)
    finally:
        ctx.lib.drg_result_free(C.byref(res))


def _blastx(s):
    ctx = _ctx()
    n_reads = len(s.nt_off) - 1
    h, n, res = C.c_void_p(), C.c_uint64(), drgpu.Result()
    ctx._check(ctx.lib.drg_batch_create_blastx(ctx.h, _p(s.nt, C.c_uint8), _p(s.nt_off, C.c_uint64), n_reads, -1,
                                               C.byref(h)))
    try:
        ctx._check(ctx.lib.drg_batch_targets(h, C.byref(n), None, None))
        ctx._check(ctx.lib.drg_batch_targets(h, C.byref(n), s.frame_query.ctypes.data_as(C.c_void_p),
                                             s.frame_index.ctypes.data_as(C.c_void_p)))
        ctx._check(ctx.lib.drg_search_batch(ctx.h, s.db.h, h, C.byref(s.cfg), C.byref(res)))
        ctx._check(ctx.lib.drg_merge_frames(C.byref(res), n_reads, _p(s.frame_query, C.c_uint32), s.cfg.max_hsps,
                                            s.cfg.max_target_seqs))
        return {**_result_columns(s, res), "frame_query": s.frame_query, "frame_index": s.frame_index}
    finally:
        ctx.lib.drg_result_free(C.byref(res))
        ctx.lib.drg_batch_destroy(h)


def run(s):
    ctx, kind = _ctx(), s.case["kind"]
    if kind == "search":
        if s.case["via"] != "requests":
            return _searched(s)
        # the served requests carry the batch's result records
        c = s.case
        serve.search_batch(ctx, s.db, s.requests, c["preset"],
                           index_chunks=None if c["chunks"] < 0 else c["chunks"])
        got = s.requests[0].raw[0]
        for buf, part in ((s.hsps, got.hsps), (s.ops, got.ops), (s.list_offsets, got.target_offsets)):
            n = min(len(buf), len(part))
            buf[:n] = part[:n]
        return _hsp_columns(s)
    if kind == "blastx":
        return _blastx(s)
    if kind == "seed_build":
        n = len(_seed_build(s.case, s.letters, s.off, s.entries))
        return {**{f: s.entries[f] for f in ("key", "seq", "pos")}, "n": n}
    if kind == "seed_join":
        out, n = C.POINTER(drgpu.SeedHit)(), C.c_uint64()
        ctx._check(ctx.lib.drg_seed_join(ctx.h, _p(s.q, drgpu.SeedEntry), len(s.q), _p(s.r, drgpu.SeedEntry),
                                         len(s.r), s.case["queries"], 4096, C.byref(out), C.byref(n)))
        _into(s.hits, out, n.value)
        ctx.lib.drg_free(out)
        return {**{f: s.hits[f] for f in ("query", "qpos", "subject", "spos")}, "n": n.value}
    seqs = (_p(s.q, C.c_uint8), _p(s.q_off, C.c_uint64), len(s.q_off) - 1, _p(s.db_letters, C.c_uint8),
            _p(s.db_off, C.c_uint64), len(s.db_off) - 1)
    n = len(s.jobs)
    if kind == "xdrop":
        out = np.empty(n, np.dtype(drgpu.Segment))
        ctx._check(ctx.lib.drg_xdrop_batch(ctx.h, *seqs, _p(s.jobs, drgpu.XdropJob), n, b"BLOSUM62", 20,
                                           _p(out, drgpu.Segment)))
        return {f: out[f] for f in ("q_start", "s_start", "len", "score")}
    matrix = s.case["matrix"].encode()
    if kind == "extend_scores":
        scores = np.empty(n, np.int32)
        ctx._check(ctx.lib.drg_extend_span_scores(ctx.h, *seqs, _p(s.jobs, drgpu.SpanJob), n, matrix, -1, -1,
                                                  _p(scores, C.c_int32), None))
        return {"score": scores}
    out = np.empty(n, np.dtype(drgpu.Aligned))
    ops, n_ops = C.POINTER(C.c_uint32)(), C.c_uint64()
    ctx._check(ctx.lib.drg_extend_span_batch(ctx.h, *seqs, _p(s.jobs, drgpu.SpanJob), n, matrix, -1, -1,
                                             _p(out, drgpu.Aligned), C.byref(ops), C.byref(n_ops)))
    _into(s.ops, ops, n_ops.value)
    ctx.lib.drg_free(ops)
    return {**{f: out[f] for f in out.dtype.names if f != "pad"}, "ops": s.ops}


# ---- what a pass cannot do without --------------------------------------------
def _mean_band(case):
    """Mean (cells, rows) of a band of _span_jobs: query length times width."""
    widths = 2 * np.array([12, 16, 30, 30, 30, 40, 64, 64]) + 1
    rng = np.random.Generator(np.random.PCG64(1))
    qlen = synth.lognormal_lengths(rng, 2000, case["q_mean"], 20, 3000)
    w = widths[np.searchsorted([50, 100, 150, 200, 250, 350, 500], qlen, side="right")]
    slen = synth.lognormal_lengths(rng, 2000, 288, 30, 5000)
    return float((np.minimum(qlen, slen) * 0.7 * w * 1.1).mean())


def work(case):
    kind = case["kind"]
    if kind in ("search", "blastx"):
        if kind == "search":
            letters = case["queries"] * case["q_mean"]
            bytes_in, hsps = letters, 4 * case["queries"]
        else:
            letters = case["reads"] * 5 * 60  # letters of the frames that keep an open reading frame
            bytes_in, hsps = case["reads"] * 225, case["reads"] // 3
        pairs = letters * case["db"] * case.get("db_mean", 288)
        cells = pairs * CELLS_PER_PAIR[case["preset"]]
        return {"bytes": bytes_in + case["db"] * case.get("db_mean", 288) + hsps * (HSP_BYTES + 40), "flops": OPS_PER_CELL * cells}
    if kind == "seed_build":
        n = case["seqs"] * case["mean"]
        return {"bytes": n + 16 * n, "flops": n * case["shape"].count("1")}
    if kind == "seed_join":
        n = case["queries"] * case["q_mean"] + case["db"] * 288
        return {"bytes": 16 * n, "flops": n}
    letters = case["queries"] * case["q_mean"] + case["db"] * 288
    if kind == "xdrop":
        # one job in five runs along a homolog for about 40 letters, the others stop within about 12
        return {"bytes": letters + case["jobs"] * (24 + 32), "flops": case["jobs"] * 18 * 3}
    cells = case["jobs"] * _mean_band(case)
    if kind == "extend_scores":
        return {"bytes": letters + case["jobs"] * (24 + 4), "flops": OPS_PER_CELL * cells}
    return {"bytes": letters + case["jobs"] * (24 + C.sizeof(drgpu.Aligned) + 40), "flops": OPS_PER_CELL * cells}


# ---- plain answers ------------------------------------------------------------
def exact(case, seed):
    """Band scores and X-drop segments, cell by cell in 64 bits; whole searches,
    seed lists and alignments have none."""
    if case["kind"] not in ("xdrop", "extend_scores") or case["jobs"] > 50000:
        return None
    s = prepare(case, seed)
    return _exact_xdrop(s) if case["kind"] == "xdrop" else {"score": _exact_scores(s)}


def _matrix(name):
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(drgpu.__file__))), "csrc", "host",
                        "score_tables.inc")
    text = open(path).read()
    at = text.index('{"%s",' % name)
    head, body = text[at:].split("\n", 2)[:2]
    vals = body[body.index("{") + 1:body.index("}")].split(",")
    gaps = [int(x) for x in head.split(",")[1:3]]
    return torch.tensor([int(v) for v in vals if v.strip()]).reshape(25, 25), gaps


def _letters_on(dev, letters, off, jobs_index):
    off = torch.from_numpy(off.astype(np.int64)).to(dev)
    at = torch.from_numpy(jobs_index.astype(np.int64)).to(dev)
    return torch.from_numpy(letters.astype(np.int64)).to(dev), off[at], off[at + 1] - off[at]


def _exact_xdrop(s):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m = _matrix("BLOSUM62")[0].to(dev)
    q, q0, qlen = _letters_on(dev, s.q, s.q_off, s.jobs["query"])
    d, s0, slen = _letters_on(dev, s.db_letters, s.db_off, s.jobs["subject"])
    qa = torch.from_numpy(s.jobs["qa"].astype(np.int64)).to(dev)
    sa = torch.from_numpy(s.jobs["sa"].astype(np.int64)).to(dev)

    def walk(score, bound, sign, first):
        st, best = score.clone(), torch.zeros_like(score)
        n = 0
        while True:
            go = (score - st < 20) & (n < bound)
            if not bool(go.any()):
                return score, best
            k = first + sign * n
            qi = (q0 + qa + k).clamp(0, len(q) - 1)
            si = (s0 + sa + k).clamp(0, len(d) - 1)
            st = torch.where(go, st + m[q[qi], d[si]], st)
            n += 1
            up = go & (st > score)
            score, best = torch.where(up, st, score), torch.where(up, n, best)
            st = torch.where(go, st, score - 20)  # a stopped walk stays stopped

    left, delta = walk(torch.zeros_like(qa), torch.minimum(qa, sa), -1, -1)
    total, length = walk(left, torch.minimum(qlen - qa, slen - sa), 1, 0)
    return {"q_start": (qa - delta).cpu().numpy(), "s_start": (sa - delta).cpu().numpy(),
            "len": (length + delta).cpu().numpy(), "score": total.cpu().numpy()}


def _exact_scores(s):
    """Banded affine Smith-Waterman (gapped.rs:67-203), rows together for all bands
    of about one width."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m, (go, ge) = _matrix(s.case["matrix"])
    m = m.to(dev)
    out = np.zeros(len(s.jobs), np.int64)
    width = (s.jobs["d1"] - s.jobs["d0"] + 1).astype(np.int64)
    order = np.argsort(width, kind="stable")
    low = -(1 << 40)
    for part in np.array_split(order, max(1, len(order) // 4000)):
        jobs = s.jobs[part]
        q, q0, qlen = _letters_on(dev, s.q, s.q_off, jobs["query"])
        d, s0, slen = _letters_on(dev, s.db_letters, s.db_off, jobs["subject"])
        d0 = torch.from_numpy(jobs["d0"].astype(np.int64)).to(dev)[:, None]
        d1 = torch.from_numpy(jobs["d1"].astype(np.int64)).to(dev)[:, None]
        w = int(width[part].max())
        x = torch.arange(w, device=dev)[None, :]  # column j = i - d1 + x
        h = torch.zeros((len(part), w + 1), dtype=torch.int64, device=dev)
        e = torch.full_like(h, low)
        h[:, w] = low
        best = torch.zeros(len(part), dtype=torch.int64, device=dev)
        for i in range(1, int(qlen.max()) + 1):
            j = i - d1 + x
            inside = (j >= 1) & (j <= slen[:, None]) & (x <= d1 - d0) & (i <= qlen[:, None])
            qi = q[(q0 + i - 1).clamp(max=len(q) - 1)][:, None]
            sc = m[qi, d[(s0[:, None] + j - 1).clamp(0, len(d) - 1)]]
            # one column to the right is the same subject column of the row above
            up_h, up_e = h[:, 1:], e[:, 1:]
            ev = torch.maximum(up_h - (go + ge), up_e - ge)
            hv = torch.maximum(torch.maximum(h[:, :-1] + sc, ev), torch.zeros_like(ev))
            hv = torch.where(inside, hv, torch.zeros_like(hv))
            run = torch.cummax(torch.where(inside, hv + ge * x, torch.full_like(hv, low)), dim=1).values
            f = torch.full_like(hv, low)
            f[:, 1:] = run[:, :-1] - go - ge * x[:, 1:]
            hv = torch.where(inside, torch.maximum(hv, f), hv)
            best = torch.maximum(best, hv.max(dim=1).values)
            h[:, :w] = torch.where(x <= d1 - d0, hv, torch.full_like(hv, low))
            e[:, :w] = torch.where(inside, ev, torch.full_like(ev, low))
        out[part] = best.cpu().numpy()
    return out
