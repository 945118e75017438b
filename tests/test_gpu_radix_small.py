"""Sorts of up to 4,096 keys, which one block does in one launch (and the
first sizes and key widths that it leaves to the passes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 63, 64, 65, 127, 129, 1438, 2048, 2049, 4095, 4096, 4097])
@pytest.mark.parametrize("begin,end", [(0, 1), (12, 64), (11, 64), (0, 52), (13, 47)])
def test_small_sorts(ctx, n, begin, end):
    r = np.random.Generator(np.random.PCG64(n * 64 + begin))
    keys = r.integers(0, 1 << 64, n, dtype=np.uint64)
    keys[r.random(n) < 0.3] = np.iinfo(np.uint64).max  # equal keys with every bit set
    sub = (keys >> np.uint64(begin)) & np.uint64((1 << (end - begin)) - 1)
    order = np.argsort(sub, kind="stable")
    k, v = ctx.radix_sort(keys, np.arange(n, dtype=np.uint32), begin, end)
    assert np.array_equal(v, order) and np.array_equal(k, keys[order])
    k, _ = ctx.radix_sort(keys, None, begin, end)
    assert np.array_equal(k, keys[order])
