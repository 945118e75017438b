"""The packed kernels take bests up to 31,743 and make a cell outside the band
dead by an addend of -16384, so a neighbour inside above that leaves it an H
above 0.  Bests of 22,000 to 27,000 over mixed letters whose path runs along a
band's edge, a few diagonals beside it, or leaves the band after a gap, in every
route of the score pass, against the oracle.  Integer work: equality."""
import numpy as np
import pytest

from drgpu import synth

pytestmark = pytest.mark.gpu
N = 2600


def _pairs(r):
    """(query, subject, diagonal before the gap, diagonal after it): three letters
    in four are W (11 against itself), a gap after 2,000 letters on either side."""
    out = []
    for gap in (0, 1, -1, 5, -5, 18, -18):
        q = np.where(r.random(N) < 0.75, 17, synth.random_protein(r, N)).astype(np.uint8)
        lead, extra = synth.random_protein(r, 7), synth.random_protein(r, abs(gap))
        if gap >= 0:  # letters of the subject without a partner
            s = np.concatenate([lead, q[:2000], extra, q[2000:]])
        else:
            s = np.concatenate([lead, q[:2000], q[2000 - gap:]])
        out.append((q, s, -7, -7 - gap))
    return out


def _jobs(pairs, width):
    jobs = []
    for k, (_, _, d, e) in enumerate(pairs):
        for off in (0, 1, 2, -1, -2):  # the lower edge, then the upper edge, beside either diagonal
            for at in {d, e}:
                jobs.append((k, k, at + off, at + off + width - 1))
                jobs.append((k, k, at + off - width + 1, at + off))
    return jobs


def _expect(orc, pairs, jobs):
    exp = [orc.extend_span(pairs[k][0], pairs[k][1], d0, d1, "BLOSUM62")[0] for k, _, d0, d1 in jobs]
    exp = [e[0] if e else 0 for e in exp]
    assert max(exp) > 22000 and all(x <= 31743 for x in exp)
    return np.array(exp)


@pytest.mark.parametrize("width", [17, 33, 151, 200, 260, 380, 500, 700, 1690])
def test_few_bands(ctx, orc, width):
    pairs = _pairs(np.random.Generator(np.random.PCG64(width)))
    jobs = _jobs(pairs, width)
    got, st = ctx.extend_span_scores([p[0] for p in pairs], [p[1] for p in pairs], jobs)
    assert sum(st["sw_class_tasks"]) == 0 and st["sw_wide_bands"] == len(jobs)
    exp = _expect(orc, pairs, jobs)
    assert np.array_equal(np.asarray(got), exp), [(jobs[k], got[k], exp[k]) for k in np.flatnonzero(got != exp)[:5]]


@pytest.mark.parametrize("width", [17, 33, 61])
def test_full_warps(ctx, orc, width):
    pairs = _pairs(np.random.Generator(np.random.PCG64(1000 + width)))
    jobs = _jobs(pairs, width)
    exp = _expect(orc, pairs, jobs)
    times = 64000 // len(jobs)
    got, st = ctx.extend_span_scores([p[0] for p in pairs], [p[1] for p in pairs], jobs * times)
    assert sum(st["sw_class_tasks"]) > 1000
    got = np.asarray(got).reshape(times, len(jobs))
    assert (got == exp).all(), [(jobs[k], got[t, k], exp[k]) for t, k in np.argwhere(got != exp)[:5]]
