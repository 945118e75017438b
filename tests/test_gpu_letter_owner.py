"""The sequence of each letter, found for 1,024 letters at a time, seen through
seed_build: sequences that end at and around the edges of a block and of a
thread's four letters, runs of empty sequences.  Against the oracle."""
import numpy as np
import pytest

from drgpu import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [
    [1024, 1024, 1023, 1, 1025, 4096],
    [1, 2, 3, 4, 5] * 300,
    [0] * 2000 + [700] + [0] * 3000 + [1500, 0, 0, 30],
    [3] * 700 + [0, 0] + [5000] + [1] * 900,
])
def test_seed_owner(ctx, orc, lengths):
    r = np.random.Generator(np.random.PCG64(len(lengths)))
    seqs = [synth.random_protein(r, n) for n in lengths]
    got = np.sort(ctx.seed_build(seqs, "1111", 0, base=3, cut=0.0), order=["key", "seq", "pos"])
    exp = np.sort(orc.seed_build(seqs, "1111", 0, base=3, cut=0.0), order=["key", "seq", "pos"])
    assert np.array_equal(got, exp)
