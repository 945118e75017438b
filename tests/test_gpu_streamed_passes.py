"""Passes that are cut because they do not fit at once: tracebacks whose trace is
above 24 GB, which reuse the trace memory batch by batch on one stream, and
index chunks whose joined hits pass the budget, which are joined one by one
after all.  Against the oracle and the uncut pass."""
import numpy as np
import pytest

import drgpu
from drgpu import synth

pytestmark = pytest.mark.gpu


def test_trace_above_the_budget(orc):
    r = np.random.Generator(np.random.PCG64(24))
    q = synth.random_protein(r, 2000)
    s = synth.random_protein(r, 4000)
    core = synth.mutate(r, q, 0.5)[:2000]
    s[900:900 + len(core)] = core
    bands = [(-2400, 599)] * 40 + [(-970, -830), (-1020, -780)]  # a block, 4 and 8 rows per lane
    jobs = [(0, 0, d0, d1) for d0, d1 in bands * 200]  # 3.3 MB of trace each of the first kind
    exp = {(d0, d1): orc.extend_span(q, s, d0, d1, "BLOSUM62")[0] for d0, d1 in set(bands)}
    ctx = drgpu.Context(0)
    try:
        got = ctx.extend_span([q], [s], jobs)
    finally:
        ctx.close()
    for k, (_, _, d0, d1) in enumerate(jobs):
        assert got[k] == exp[d0, d1], k


@pytest.mark.parametrize("index", [0, 4 << 30])
def test_joined_hits_above_the_budget(ctx, index):
    w = synth.workload(2, n_queries=1600, n_db=7860, seed_offset=9)
    dl, do = drgpu.concat(w.db)
    tl, to = drgpu.concat(w.queries)
    res = drgpu.ResidentDb(ctx, dl, do, index_budget=index)
    b = drgpu.ResidentBatch(ctx, tl, to)
    try:
        out = []
        for budget in (0, 1 << 24, 1 << 24):
            cfg = drgpu.make_config(sensitivity="very-sensitive", index_chunks=4, max_hits_per_pass=budget)
            lists, st, _ = drgpu.search_resident(ctx, res, b, cfg)
            out.append(([[h.key() for h in lst] for lst in lists], st))
            assert st["hits"] > 1 << 24
    finally:
        b.close()
        res.close()
    whole, st0 = out[0]
    assert st0["hit_passes"] == 1 and sum(map(len, whole)) > 0
    for got, st in out[1:]:
        assert st["hit_passes"] > 1
        assert got == whole
        for k in ("hits", "ref_seeds", "unique_hits", "bands", "hsps"):
            assert st[k] == st0[k], k
