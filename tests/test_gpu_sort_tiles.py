"""The radix sort around its two tile sizes (512 items a warp below 4,194,304 items, else 2048) and the one-block scan's
limit (65,536 counts, 131,072 items), against numpy's stable sort."""
import numpy as np
import pytest

from tests.test_gpu_sort import _sort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [511, 512, 513, 131_071, 131_072, 131_073, 131_585, 4_194_303, 4_194_304, 4_194_305])
def test_around_the_tile_sizes(cuda_device, n):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 27, n, dtype=np.uint32)
    keys[rng.random(n) < 0.5] &= np.uint32(0x7000003)
    vals = np.arange(n, dtype=np.uint32)
    ko, vo = _sort(keys, vals, 0, 27)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(vo, vals[order]) and np.array_equal(ko, keys[order])
