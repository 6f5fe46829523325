"""The radix sort of a queue whose length only the device knows (the wavefront's ray order): the first *count items are
sorted as numpy's stable sort does, nothing behind them is written, and a queue of `above` items or fewer is left
alone. Lengths around the tile sizes, the threshold and the capacity."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests.test_gpu_sort import LIB

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,above,counts", [
    (5000, 0, (0, 1, 31, 511, 512, 513, 2049, 4999, 5000, 6000)),
    (200_000, 131_072, (1, 131_071, 131_072, 131_073, 131_585, 199_999, 200_000)),
    (4_194_400, 131_072, (131_072, 131_073, 133_121, 4_194_303, 4_194_400)),
])
def test_counted_sort(cuda_device, n, above, counts):
    lib = C.CDLL(LIB)
    lib.ptirkat_radix_sort_counted.argtypes = [C.c_int] + [C.c_void_p] * 4 + [C.c_longlong, C.c_int, C.c_int, C.c_void_p,
                                                                             C.c_uint]
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 27, n, dtype=np.uint32)
    keys[rng.random(n) < 0.3] &= np.uint32(0x7000003)
    vals = np.arange(n, dtype=np.uint32)
    ki, vi = (torch.from_numpy(a.view(np.int32).copy()).cuda() for a in (keys, vals))
    for count in counts:
        ko, vo = torch.full_like(ki, -1), torch.full_like(vi, -1)
        c = torch.tensor([count], dtype=torch.int32, device=cuda_device)
        rc = lib.ptirkat_radix_sort_counted(4, ki.data_ptr(), ko.data_ptr(), vi.data_ptr(), vo.data_ptr(), n, 0, 27,
                                            c.data_ptr(), above)
        assert rc == 0
        m = min(count, n) if count > above else 0
        order = np.argsort(keys[:m], kind="stable")
        k, v = ko.cpu().numpy().view(np.uint32), vo.cpu().numpy().view(np.uint32)
        assert np.array_equal(k[:m], keys[order]) and np.array_equal(v[:m], vals[order]), count
        assert (k[m:] == 0xFFFFFFFF).all() and (v[m:] == 0xFFFFFFFF).all(), count
