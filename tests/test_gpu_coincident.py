"""Gaussians cloned in place (one position, rotation, scale and density; albedo and SH of their own) among others:
small launches, four lanes a ray, against the megakernel. With sixteen Gaussians one round holds every candidate,
so both insert the same candidates in the same order. A lost or doubled Gaussian moves the material by
its weight, of order 0.1, and the flags; equal buffers leave the rounding of two compilations of the same sums, below
1e-5 of values up to 1, and for a gradient summed by atomics over the rays 1e-4 of the largest."""
import numpy as np
import pytest
import torch

from tests.scenes import gpu_trace, gpu_trace_bwd, make_tracer, small_scene, to_torch

pytestmark = pytest.mark.gpu


def _scene(copies, others, seed):
    n = copies + others
    s = small_scene(n=n, w=40, h=30, spp=1, max_bounces=1, seed=seed, scale_range=(0.3, 0.9), sh_full=True)
    rng = np.random.default_rng(seed)
    who = rng.permutation(n)[:copies]
    for k in ("build_pos", "build_rot", "build_scl", "build_dns", "density"):
        s[k][who] = s[k][who[0]]
    s["build_dns"][:] = 0.05 + 0.15 * s["build_dns"]
    s["density"][:, 3] = s["build_dns"][:, 0]
    return s


@pytest.mark.parametrize("copies", [1, 4, 5, 6, 8, 12])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_clones_match_the_megakernel(cuda_device, copies, seed):
    S = to_torch(_scene(copies, 16 - copies, seed))
    got = []
    for schedule in ("wavefront", "megakernel"):
        tr = make_tracer(clamping=False, mis=False, schedule=schedule)
        fwd = gpu_trace(tr, S)
        torch.manual_seed(3)
        _, mg, _, _, _ = gpu_trace_bwd(tr, S, fwd, torch.zeros_like(fwd[10]), material_grad=torch.randn_like(fwd[7]))
        torch.cuda.synchronize()
        assert tr.device_status() == 0
        got.append([fwd[i].clone() for i in (0, 1, 2, 7, 8, 9)] + [mg])
    (*a, ma), (*b, mb) = got
    assert torch.equal(a[5], b[5])  # visibility
    assert torch.equal(a[4], b[4])  # hit counts
    for x, y in zip(a[:4], b[:4]):
        assert float((x - y).abs().max()) <= 1e-5 * max(1.0, float(y.abs().max()))
    assert float((ma - mb).abs().max()) <= 1e-4 * float(mb.abs().max())
