"""The order in which a traversal visits the children of a node, shown by clones of one Gaussian (albedo of their own):
every box entry and every candidate's distance is equal, so a round of sixteen composites, and the adjoint's replay
scatters to, the first candidates that the visits come to. One lane a ray (180,000 rays) and four (600) against
the megakernel, which has the order of descend (traverse.cuh). Other candidates, or another order, move the
material by their weights, of order 0.1; equal order leaves the rounding of two compilations of the same sums, below
1e-5 of values up to 1, and for a gradient summed by atomics over the rays 1e-4 of the largest."""
import pytest
import torch

from tests.scenes import gpu_trace, gpu_trace_bwd, make_tracer, small_scene, to_torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(30, 20), (450, 400)])
@pytest.mark.parametrize("n", [17, 40, 200])
def test_clones_come_in_descend_order(cuda_device, w, h, n):
    s = small_scene(n=n, w=w, h=h, spp=1, max_bounces=1, seed=n)
    for name in ("build_pos", "build_rot", "build_scl", "build_dns", "density"):
        s[name][:] = s[name][:1]
    s["build_scl"][:] = s["density"][:, 8:11] = 0.4
    s["build_dns"][:] = s["density"][:, 3:4] = 0.1
    S = to_torch(s)
    got = []
    for schedule in ("wavefront", "megakernel"):
        tr = make_tracer(clamping=False, mis=False, schedule=schedule)
        fwd = gpu_trace(tr, S)
        torch.manual_seed(3)
        _, mg, _, _, _ = gpu_trace_bwd(tr, S, fwd, torch.zeros_like(fwd[10]), material_grad=torch.randn_like(fwd[7]))
        torch.cuda.synchronize()
        assert tr.device_status() == 0
        got.append((fwd[7].clone(), fwd[8].clone(), fwd[9].clone(), mg))
    (ma, ha, va, ga), (mb, hb, vb, gb) = got
    assert float(hb.max()) == 16 and torch.equal(ha, hb) and torch.equal(va, vb)
    assert float((ma - mb).abs().max()) <= 1e-5
    assert float((ga - gb).abs().max()) <= 1e-4 * float(gb.abs().max())
