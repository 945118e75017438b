"""The 32-bit systolic DP (tracebacks, and scores of bands the packed kernels
leave) against the oracle, at the edges of its routes: 4 rows per lane up to
151 columns, 8 rows up to 271 (tracebacks), a block per band above; strips of
4, 8 and 128 rows; bands partly or wholly off the matrix; rows past the
subject's end.  Integer work: equality."""
import numpy as np
import pytest

from drgpu import synth

pytestmark = pytest.mark.gpu


def _related(r, n, m):
    """A query and a subject that share a mutated core, so that bands hold alignments."""
    q = synth.random_protein(r, n)
    core = synth.mutate(r, q, 0.6)[:m]
    s = synth.random_protein(r, m)
    at = int(r.integers(0, m - len(core) + 1))
    s[at:at + len(core)] = core
    return q, s


def _check(ctx, orc, qs, ss, jobs, matrix="BLOSUM62"):
    got = ctx.extend_span(qs, ss, jobs, matrix)
    scores, _ = ctx.extend_span_scores(qs, ss, jobs, matrix)
    for k, (a, b, d0, d1) in enumerate(jobs):
        exp, _ = orc.extend_span(qs[a], ss[b], d0, d1, matrix)
        assert got[k] == exp, (k, len(qs[a]), len(ss[b]), d0, d1)
        assert int(scores[k]) == (exp[0] if exp else 0), (k, len(qs[a]), len(ss[b]), d0, d1)


@pytest.mark.parametrize("width", [1, 2, 5, 16, 17, 33, 129, 150, 151, 152, 153, 270, 271, 272, 600])
def test_widths(ctx, orc, width):
    r = np.random.Generator(np.random.PCG64(width))
    qs, ss, jobs = [], [], []
    for n, m in ((1, 40), (3, 7), (4, 200), (5, 5), (8, 300), (127, 129), (128, 64), (129, 400), (257, 256), (500, 333)):
        q, s = _related(r, n, m)
        qs.append(q)
        ss.append(s)
        i = len(qs) - 1
        # centred, at either edge, wholly off the matrix on each side, past the subject's end
        for mid in (0, n // 2, -m // 2, n + width, -m - width, n - m, m // 3):
            jobs.append((i, i, mid - width // 2, mid - width // 2 + width - 1))
    _check(ctx, orc, qs, ss, jobs, "BLOSUM62" if width % 2 else "BLOSUM45")


@pytest.mark.parametrize("n,m,width", [(1300, 1200, 1701), (2100, 900, 2900), (700, 2500, 3000), (1025, 1025, 850),
                                       (2900, 2950, 129), (129, 3000, 2 * 10 ** 9)])
def test_long_and_wide(ctx, orc, n, m, width):
    r = np.random.Generator(np.random.PCG64(n + m))
    q, s = _related(r, n, m)
    d = (n - m) // 2
    _check(ctx, orc, [q], [s], [(0, 0, d - width // 2, d - width // 2 + width - 1), (0, 0, -5, 5 + width // 3)])


def test_saturating_score(ctx, orc):
    # an identical pair whose score passes 2^15: never the packed kernels'
    q = np.full(3100, 17, np.uint8)  # W scores 11
    _check(ctx, orc, [q], [q.copy()], [(0, 0, -12, 12), (0, 0, -150, 150), (0, 0, -400, 3000)])


def test_many_bands_of_mixed_routes(ctx, orc):
    r = np.random.Generator(np.random.PCG64(5))
    qs, ss = zip(*[_related(r, int(n), int(m)) for n, m in zip(r.integers(20, 400, 24), r.integers(400, 600, 24))])
    jobs = [(k % 24, k % 24, int(c) - int(w) // 2, int(c) - int(w) // 2 + int(w) - 1)
            for k, (w, c) in enumerate(zip(r.integers(1, 420, 240), r.integers(-300, 200, 240)))]
    _check(ctx, orc, list(qs), list(ss), jobs, "PAM70")


def test_two_bands_per_warp(ctx, orc):
    # the score pass's lane kernel: the edges of its three widths, an odd count,
    # halves of a warp of very different lengths, a best just below 0x7C00
    r = np.random.Generator(np.random.PCG64(77))
    qs, ss = zip(*[_related(r, n, m) for n, m in ((1, 30), (3, 60), (33, 40), (300, 280), (640, 600), (1100, 1500))])
    qs, ss = list(qs), list(ss)
    jobs = [(k, k, -w // 2, -w // 2 + w - 1) for w in (17, 18, 31, 136, 137, 151, 152, 271, 272, 273, 511, 512)
            for k in range(6)]
    jobs.append((5, 5, -60, 60))
    _check(ctx, orc, qs, ss, jobs)
    q = np.full(2885, 17, np.uint8)  # W scores 11: 31,735
    _check(ctx, orc, [q, qs[2]], [q.copy(), ss[2]], [(0, 0, -10, 10), (1, 1, -10, 10), (0, 0, -250, 250)])
