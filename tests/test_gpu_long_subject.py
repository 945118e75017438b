"""The block kernel of the 32-bit DP keeps a row per block as long as the
longest subject, so with a long one fewer rows than blocks fit its memory: more
bands than rows, each of more than eight strips of 128 rows (the rows are read
there), on subjects of 100,400 and 4.2M letters, beside bands on short ones of
the same set, and with the long one in the set alone.  Against the oracle."""
import numpy as np
import pytest

from drgpu import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,on_long,others", [(100_400, 300, 130), (4_200_000, 10, 20), (4_200_000, 0, 40)])
def test_more_bands_than_rows(ctx, orc, m, on_long, others):
    r = np.random.Generator(np.random.PCG64(m + on_long))
    qs = [synth.random_protein(r, int(n)) for n in r.integers(910, 1200, 12)]
    long = synth.random_protein(r, m)
    ss, jobs = [long], []
    for k in range(on_long):
        q = qs[k % len(qs)]
        core = synth.mutate(r, q, 0.5)
        at = (m - 1500) * k // max(1, on_long - 1) if m > 1_000_000 else int(r.integers(0, m - len(core)))
        long[at:at + len(core)] = core
        w = int(r.integers(280, 420)) if k % 5 else 1750
        jobs.append((k % len(qs), 0, -at - w // 2, -at + w // 2))
    for k in range(others):
        q = qs[k % len(qs)]
        s = synth.random_protein(r, int(r.integers(1000, 1400)))
        core = synth.mutate(r, q, 0.5)[:len(s)]
        s[:len(core)] = core
        ss.append(s)
        w = int(r.integers(280, 420))
        jobs.append((k % len(qs), len(ss) - 1, -w // 2, w // 2))
    got = ctx.extend_span(qs, ss, jobs)
    scores, _ = ctx.extend_span_scores(qs, ss, jobs)
    for k, (a, b, d0, d1) in enumerate(jobs):
        exp, _ = orc.extend_span(qs[a], ss[b], d0, d1, "BLOSUM62")
        assert got[k] == exp, (k, d0, d1)
        assert int(scores[k]) == exp[0], (k, d0, d1)
