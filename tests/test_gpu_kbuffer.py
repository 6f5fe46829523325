"""The k-buffer in all its forms (one lane a ray with ids in registers, spread over four lanes with and without the
entry pushed out, distances alone with a log of ids) against the sorted insertion written out: a new entry
goes behind equal distances, and what it displaces moves on behind everything at its own distance. Runs of equal
distances of every length up to the buffer's and past it, among other distances in any order. All values equal."""
import ctypes as C
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LIB = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle", "libptir_kat.so")
FAR, NONE = np.float32(1e20), 0xFFFFFFFF
CASES, M = 301, 40


def _chain(k, ts, ids):
    """(distances, ids, id pushed out by each insertion) of one sequence."""
    kt, kid, out = [FAR] * k, [NONE] * k, []
    for t, i in zip(ts, ids):
        if not t < kt[-1]:
            out.append(NONE)
            continue
        for j in range(k):
            if t < kt[j]:
                kt[j], t = t, kt[j]
                kid[j], i = i, kid[j]
        out.append(i)
    return kt, kid, out


def _sequences(run):
    """CASES sequences of M distances: `run` at one distance among others, or few distances over and over."""
    rng = np.random.default_rng(run)
    ts = rng.uniform(0.5, 4.0, (CASES, M)).astype(np.float32)
    for row in ts[:CASES // 2]:
        row[rng.permutation(M)[:run]] = np.float32(rng.uniform(0.5, 4.0))
    ts[CASES // 2:] = rng.integers(1, 2 + 40 // run, (CASES - CASES // 2, M)).astype(np.float32)
    ids = np.stack([rng.permutation(M) for _ in range(CASES)]).astype(np.uint32)
    return ts, ids


@pytest.mark.parametrize("k", [8, 16])
@pytest.mark.parametrize("run", [1, 2, 3, 4, 5, 6, 8, 12, 17, 33])
def test_forms_agree_with_the_chain(cuda_device, k, run):
    lib = C.CDLL(LIB)
    lib.ptirkat_kbuffer.argtypes = [C.c_int] * 4 + [C.c_void_p] * 5
    ts, ids = _sequences(run)
    want = [_chain(k, t, i) for t, i in zip(ts, ids)]
    wt, wid, wev = (np.array([w[j] for w in want], dt) for j, dt in ((0, np.float32), (1, np.uint32), (2, np.uint32)))
    dt, di = (torch.from_numpy(a.copy()).cuda() for a in (ts, ids.view(np.int32)))
    for form in range(4):
        ot = torch.zeros((CASES, k), device=cuda_device)
        oi, ev = (torch.zeros((CASES, n), dtype=torch.int32, device=cuda_device) for n in (k, M))
        rc = lib.ptirkat_kbuffer(k, form, CASES, M, dt.data_ptr(), di.data_ptr(), ot.data_ptr(), oi.data_ptr(), ev.data_ptr())
        assert rc == 0
        assert np.array_equal(ot.cpu().numpy(), wt), form
        assert np.array_equal(oi.cpu().numpy().view(np.uint32), wid), form
        if form in (0, 2):
            assert np.array_equal(ev.cpu().numpy().view(np.uint32), wev), form
