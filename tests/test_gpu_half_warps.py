"""The packed score kernel runs two tasks per warp, each of up to 16 bands of
one query window (or one subject): task sizes around 16, odd counts of tasks,
partners of different lengths, widths and orientation, against the lane
kernel on every band and the oracle on some.  Integer work: equality."""
import numpy as np
import pytest

from drgpu import synth

pytestmark = pytest.mark.gpu


def _bands(seed, sizes, widths, n_mean, m_mean):
    """Groups of `sizes` bands per query; enough bands that whole warps stay with the packed kernel."""
    r = np.random.Generator(np.random.PCG64(seed))
    ss = [synth.random_protein(r, max(20, int(v))) for v in r.gamma(6, m_mean / 6, 400)]
    qs, jobs = [], []
    for g in sizes:
        n = max(17, int(r.gamma(6, n_mean / 6)))
        q = synth.random_protein(r, n)
        qs.append(q)
        for t in range(g):
            b = int(r.integers(0, len(ss)))
            if t % 5 == 0:  # some of them related
                core = synth.mutate(r, q, 0.7)[:len(ss[b])]
                ss[b][:len(core)] = core
            w = int(r.choice(widths))
            d = int(r.integers(-len(ss[b]) + 1, n)) - w // 2
            jobs.append((len(qs) - 1, b, d, d + w - 1))
    return qs, ss, jobs


@pytest.mark.parametrize("widths,n_mean,m_mean", [
    ([33], 60, 60),                          # one width: unrolled epilogue
    ([17, 18, 33, 64, 129, 136], 90, 70),    # mixed widths of one class
    ([129, 137, 200, 272], 120, 150),        # two classes
    ([129], 400, 60),                        # subjects as rows
])
def test_task_pairs(ctx, orc, widths, n_mean, m_mean):
    sizes = [1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 5] * 160
    qs, ss, jobs = _bands(len(widths) + n_mean, sizes, widths, n_mean, m_mean)
    got, st = ctx.extend_span_scores(qs, ss, jobs)
    assert sum(st["sw_class_tasks"]) > 200
    exp = []
    for at in range(0, len(jobs), 500):  # calls too small to fill warps: the lane kernel
        e, st = ctx.extend_span_scores(qs, ss, jobs[at:at + 500])
        assert sum(st["sw_class_tasks"]) == 0
        exp.extend(e)
    bad = np.flatnonzero(np.asarray(got) != np.asarray(exp))
    assert len(bad) == 0, [(jobs[k], int(got[k]), int(exp[k])) for k in bad[:5]]
    r = np.random.Generator(np.random.PCG64(1))
    for k in r.choice(len(jobs), 200, replace=False):
        a, b, d0, d1 = jobs[k]
        e, _ = orc.extend_span(qs[a], ss[b], d0, d1, "BLOSUM62")
        assert int(got[k]) == (e[0] if e else 0), jobs[k]
