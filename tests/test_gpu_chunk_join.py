"""Index chunks joined together: the expansion cap counts reference
occurrences per chunk (search.rs:127-131), so a search's hits depend on the
chunk count; one joined pass, one pass per chunk (more than 16 chunks, or a
small hit budget) and cached chunk indexes give the oracle's answer."""
import numpy as np
import pytest

import drgpu
from drgpu import synth

pytestmark = pytest.mark.gpu


def _keys(lists):
    return [[h.key() for h in lst] for lst in lists]


@pytest.fixture(scope="module")
def workload():
    # a motif in 60 queries and 90 sequences, unevenly along the database: its
    # keys pass the cap whole, and in some chunks of a split only
    r = np.random.Generator(np.random.PCG64(99))
    motif = synth.random_protein(r, 24)

    def with_motif(n):
        s = synth.random_protein(r, n)
        at = int(r.integers(0, n - 24))
        s[at:at + 24] = motif
        return s

    queries = [with_motif(int(n)) for n in r.integers(100, 300, 60)]
    db = [with_motif(int(n)) for n in r.integers(80, 400, 70)] + \
        [synth.random_protein(r, int(n)) for n in r.integers(30, 300, 60)] + \
        [with_motif(int(n)) for n in r.integers(80, 400, 20)] + [np.zeros(0, np.uint8)]
    return queries, db


@pytest.mark.parametrize("sens", ["fast", "default", "sensitive", "very-sensitive"])
@pytest.mark.parametrize("chunks", [1, 2, 4, 7, 16, 17])
def test_chunk_counts(ctx, orc, workload, sens, chunks):
    queries, db = workload
    dl, do = drgpu.concat(db)
    tl, to = drgpu.concat(queries)
    exp, _ = orc.search(db, queries, sensitivity=sens, index_chunks=chunks, threads=8)
    got, st = ctx.search(dl, do, tl, to, drgpu.make_config(sensitivity=sens, index_chunks=chunks))
    assert _keys(got) == exp
    small, st2 = ctx.search(dl, do, tl, to, drgpu.make_config(sensitivity=sens, index_chunks=chunks,
                                                             max_hits_per_pass=5000))
    assert _keys(small) == exp
    for k in ("hits", "ref_seeds", "unique_hits", "bands"):
        assert st[k] == st2[k], k
    # per chunk the cap lets pairs through that the whole database's count rejects
    if chunks >= 4:
        whole, _ = ctx.search(dl, do, tl, to, drgpu.make_config(sensitivity=sens, index_chunks=1))
        assert _keys(whole) != exp


@pytest.mark.parametrize("requests", [False, True])
def test_cached_chunks(ctx, orc, workload, requests):
    queries, db = workload
    dl, do = drgpu.concat(db)
    tl, to = drgpu.concat(queries)
    rid = np.repeat(np.arange(6), 10).astype(np.uint32)
    exp = []
    for k in range(6) if requests else [None]:
        part = queries if k is None else queries[10 * k:10 * k + 10]
        e, _ = orc.search(db, part, sensitivity="default", index_chunks=4, threads=8)
        exp += [[(h[0] + (0 if k is None else 10 * k),) + tuple(h[1:]) for h in lst] for lst in e]
    res = drgpu.ResidentDb(ctx, dl, do, index_budget=1 << 30)
    b = drgpu.ResidentBatch(ctx, tl, to, request=rid if requests else None)
    try:
        for hits in (0, 4):  # built, then read
            lists, st, _ = drgpu.search_resident(ctx, res, b, drgpu.make_config(sensitivity="default", index_chunks=4))
            assert [[tuple(h.key()) for h in lst] for lst in lists] == exp
            assert st["index_hits"] == hits
        s = res.index_stats()
        assert s["hits"] == 4 and s["misses"] == 4
    finally:
        b.close()
        res.close()
