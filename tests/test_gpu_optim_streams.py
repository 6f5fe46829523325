"""Two fused Adam steps over one parameter, each of the rows that the other hides, on two streams at a time: a step
writes no element of a hidden row, so every row ends as after its own steps alone, bit for bit. Rows whose
borders lie within a group of four elements, and rows whose borders do not."""
import pytest
import torch

from ptir_b200.optim import selective_adam_

pytestmark = pytest.mark.gpu

N, STEPS = 200_000, 40


def _run(row, apart):
    g = torch.Generator(device="cuda").manual_seed(row)
    p, grad, m, v = (torch.randn((N, row), generator=g, device="cuda") for _ in range(4))
    v.abs_()
    odd = torch.arange(N, device="cuda") % 2
    sides = [(odd == k).to(torch.uint8) for k in (0, 1)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in sides] if apart else [torch.cuda.current_stream()] * 2
    for _ in range(STEPS):
        for vis, s in zip(sides, streams):
            with torch.cuda.stream(s):
                selective_adam_(p, grad, m, v, vis, 1e-2)
    torch.cuda.synchronize()
    return p, m, v


@pytest.mark.parametrize("row", [1, 3, 4, 5, 27])
def test_steps_of_other_rows_on_two_streams(cuda_device, row):
    for a, b in zip(_run(row, True), _run(row, False)):
        assert torch.equal(a, b)
