"""The lane kernel of the score pass at the widest bands that its lanes hold:
a lane turns to its next strip right after the strip of 32 before passed its
last column, beside strips that still run.  Low-complexity sequences, so that
any value that crosses a band's edge changes a score.  Against the oracle."""
import numpy as np
import pytest

from drgpu import synth

pytestmark = pytest.mark.gpu

ROWS = [4, 6, 8, 12, 16]
WIDEST = [31 * (r + 1) - r for r in ROWS]


@pytest.mark.parametrize("width", [w - d for w in WIDEST for d in (0, 1, 2, 3, 5, 9, 17)] + [w + 1 for w in WIDEST])
def test_widest_bands(ctx, orc, width):
    r = np.random.Generator(np.random.PCG64(width))
    qs, ss, jobs = [], [], []
    for n, m in ((260, 700), (700, 260), (900, 900), (1300, 1000)):
        for kind in range(3):
            if kind == 0:  # one letter everywhere
                q, s = np.full(n, 17, np.uint8), np.full(m, 17, np.uint8)
            elif kind == 1:  # long runs
                q = np.repeat(synth.random_protein(r, n // 10 + 1), 10)[:n]
                s = np.repeat(synth.random_protein(r, m // 10 + 1), 10)[:m]
            else:
                q, s = synth.random_protein(r, n), synth.random_protein(r, m)
                s[:min(n, m)] = q[:min(n, m)]
            qs.append(q)
            ss.append(s)
            for mid in (0, 40, -40, n // 3, -m // 3, n - m // 2):
                jobs.append((len(qs) - 1, len(ss) - 1, mid - width // 2, mid - width // 2 + width - 1))
    got, _ = ctx.extend_span_scores(qs, ss, jobs)
    for k, (a, b, d0, d1) in enumerate(jobs):
        e, _ = orc.extend_span(qs[a], ss[b], d0, d1, "BLOSUM62")
        assert int(got[k]) == (e[0] if e else 0), jobs[k]


@pytest.mark.parametrize("rows,width", [(8191, 151), (8192, 200), (8193, 200), (16384, 100), (16385, 100)])
def test_longest_traced_bands(ctx, orc, rows, width):
    # at the row limit of the rotating traceback kernel the block kernel takes over
    r = np.random.Generator(np.random.PCG64(rows))
    q = synth.random_protein(r, rows)
    s = synth.mutate(r, q, 0.8)
    jobs = [(0, 0, -width // 2, -width // 2 + width - 1)]
    got = ctx.extend_span([q], [s], jobs)
    exp, _ = orc.extend_span(q, s, jobs[0][2], jobs[0][3], "BLOSUM62")
    assert got[0] == exp
