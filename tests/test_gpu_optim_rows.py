"""The fused Adam step over row lengths and counts around its groups of four elements, aligned and not, against the
same update in numpy float32 (the operations are IEEE float32 in one order up to the contraction of b1 m + (1 - b1) g
and b2 v + (1 - b2) g g, one rounding each: two ulp of the moments, and of a step of at most lr / sqrt(1 - b2))."""
import numpy as np
import pytest
import torch

from ptir_b200.optim import SelectiveAdam, selective_adam_

pytestmark = pytest.mark.gpu


def _expect(p, g, m, v, vis, lr, b1, b2, eps):
    f = np.float32
    on = np.ones(len(p), bool) if vis is None else vis != 0
    m2 = f(b1) * m + (f(1) - f(b1)) * g
    v2 = f(b2) * v + (f(1) - f(b2)) * g * g
    p2 = p - f(lr) * m2 / (np.sqrt(v2) + f(eps))
    on = on.reshape(-1, *([1] * (p.ndim - 1)))
    return np.where(on, p2, p), np.where(on, m2, m), np.where(on, v2, v)


@pytest.mark.parametrize("row", [1, 2, 3, 4, 5, 7, 48])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 257, 1030])
@pytest.mark.parametrize("visible", [None, "some", "none"])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows(cuda_device, row, n, visible, shift):
    rng = np.random.default_rng(row * 100 + n)
    a = [rng.standard_normal((n, row)).astype(np.float32) for _ in range(3)]
    a.append(rng.uniform(0, 1, (n, row)).astype(np.float32))  # param, grad, m, v
    vis = None if visible is None else (rng.random(n) < (0.5 if visible == "some" else 0.0)).astype(np.uint8)
    bufs = []
    for x in a:  # `shift` elements off a 16-byte boundary
        b = torch.full((n * row + 8,), 7.0, device=cuda_device)
        b[shift:shift + n * row] = torch.from_numpy(x.reshape(-1)).to(cuda_device)
        bufs.append(b)
    view = [b[shift:shift + n * row].view(n, row) for b in bufs]
    tv = None if vis is None else torch.from_numpy(vis).to(cuda_device)
    selective_adam_(view[0], view[1], view[2], view[3], tv, 1e-2, 0.9, 0.999, 1e-8)
    want = _expect(a[0], a[1], a[2], a[3], vis, 1e-2, 0.9, 0.999, 1e-8)
    for got, w in zip((view[0], view[2], view[3]), want):
        np.testing.assert_allclose(got.cpu().numpy(), w, rtol=1e-6, atol=1e-6)
    hidden = slice(None) if visible == "none" else (None if vis is None else torch.from_numpy(vis == 0))
    if hidden is not None:  # hidden rows bit for bit
        for got, x in zip((view[0], view[2], view[3]), (a[0], a[2], a[3])):
            assert torch.equal(got.cpu()[hidden], torch.from_numpy(x)[hidden])
    for b in bufs:  # nothing written around the buffers
        assert bool((b[:shift] == 7.0).all()) and bool((b[shift + n * row:] == 7.0).all())


def test_groups_share_their_flags(cuda_device):
    g = torch.Generator().manual_seed(2)
    ps = [torch.nn.Parameter(torch.randn(s, generator=g).to(cuda_device)) for s in ((40, 5), (40, 48), (30, 3))]
    before = [p.detach().clone() for p in ps]
    for p in ps:
        p.grad = torch.ones_like(p)
    vis = (torch.arange(40, device=cuda_device) % 3 == 0).float().reshape(40, 1)
    SelectiveAdam([{"params": [p], "lr": 0.1} for p in ps]).step(vis)
    for p, b in zip(ps, before):
        moved = (p.detach() != b).any(1)
        assert torch.equal(moved, vis.reshape(-1)[:len(p)] != 0)
