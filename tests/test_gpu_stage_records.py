"""seed::build and seed::join_into records made on the device, against the
oracle: key widths on both sides of 32 bits, empty sequences, empty inputs,
hit keys of more than 64 bits."""
import numpy as np
import pytest

from drgpu import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,reduction", [("1", 1), ("111111111", 0), ("1" * 10, 1), ("1" * 9, 0), ("1" * 10, 0),
                                             ("1111111", 2), ("11111111", 2), ("1" * 14, 2), ("1" * 15, 2),
                                             ("1" * 16, 2)])
def test_seed_entries(ctx, orc, shape, reduction):
    # key bits run from 4 to beyond 64 (20^16 wraps); equal keys stay in letter order
    r = np.random.Generator(np.random.PCG64(len(shape) + reduction))
    seqs = [synth.random_protein(r, int(n)) for n in (0, 300, 0, 0, 17, 1, 255, 256, 0)]
    seqs[1][100:200] = seqs[1][0:100]
    got = ctx.seed_build(seqs, shape, reduction, base=5, cut=0.0)
    exp = orc.seed_build(seqs, shape, reduction, base=5, cut=0.0)
    assert len(got) == len(exp)
    assert (got == np.sort(exp, order=["key", "seq", "pos"])).all()


@pytest.mark.parametrize("seqs", [[], [np.zeros(0, np.uint8)] * 3, [np.full(2, 3, np.uint8)]])
def test_no_seeds(ctx, seqs):
    assert len(ctx.seed_build(seqs, "1111", 0, base=0, cut=0.0)) == 0
