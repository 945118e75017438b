"""Six-frame translation a warp per frame: frames that end at and around 32
codons, stop-free stretches that begin and end in different groups of 32 or
are just as long as the limit.  Against the oracle, byte for byte."""
import numpy as np
import pytest

from test_gpu_blastx import oracle_frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("min_orf", [-1, 2, 31, 32, 33, 64, 65, 500])
def test_frame_groups(ctx, orc, min_orf):
    r = np.random.Generator(np.random.PCG64(900 + min_orf))
    reads = ["".join(r.choice(list("ACGT"), size=n)) for n in
             [93, 94, 95, 96, 97, 98, 99, 189, 192, 195, 287, 288, 289, 290, 960, 3001]]
    for gap in (1, 31, 32, 33, 63, 64, 65, 100):  # stops that far apart, in frame 0 and on the other strand
        reads.append("ATG" + ("GCA" * (gap - 1) + "TAA") * 7 + "GCC" * 40)
        reads.append("GGC" * 35 + ("TTA" + "TGC" * (gap - 1)) * 6)
    got, q, f = ctx.translate_reads(reads, min_orf)
    exp, eq, ef = oracle_frames(orc, reads, min_orf)
    assert list(q) == eq and list(f) == ef
    assert len(got) == len(exp) and all(np.array_equal(a, b) for a, b in zip(got, exp))
