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


def _entries(r, keys, n, seqs, poss):
    e = np.zeros(n, dtype=[("key", "u8"), ("seq", "u4"), ("pos", "u4")])
    e["key"] = np.sort(r.choice(keys, n))
    e["seq"] = r.choice(seqs, n)
    e["pos"] = r.choice(poss, n)
    return e


@pytest.mark.parametrize("seqs,poss", [
    ([0], [0]),                                    # every field zero bits wide
    ([0, 1, 70], [0, 1, 5, 1000]),
    ([3, 2 ** 20], [0, 2 ** 20 - 1]),              # exactly 64 bits: 2 + 21 + 21 + 20
    ([3, 2 ** 20], [0, 2 ** 20]),                  # 66
    ([7, 2 ** 32 - 1], [0, 2 ** 31, 2 ** 32 - 1]),  # 99
])
def test_join_records(ctx, orc, seqs, poss):
    r = np.random.Generator(np.random.PCG64(len(seqs) + len(poss)))
    keys = np.array([0, 3, 4, 2 ** 40, 2 ** 64 - 1], np.uint64)
    q = _entries(r, keys, 40, [0, 2, 3], poss)
    e = _entries(r, keys, 90, seqs, poss)
    for cap in (4096, 150):
        assert ctx.seed_join(q, e, 4, cap) == orc.seed_join(q, e, 4, cap)


def test_join_rejects_a_target_out_of_range(ctx):
    import drgpu
    r = np.random.Generator(np.random.PCG64(1))
    q = _entries(r, np.array([1], np.uint64), 3, [4], [0])
    with pytest.raises(drgpu.DrgError) as e:
        ctx.seed_join(q, q, 4)
    assert e.value.code == 1
    assert ctx.seed_join(q[:0], q, 4) == [] and ctx.seed_join(q, q[:0], 5) == []
