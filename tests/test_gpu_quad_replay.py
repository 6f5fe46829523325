"""The adjoint's re-traversals, four lanes a job (resumed rounds, up to 131,072 jobs) against one lane a job from the
root (resume_rounds=1). Both visit a segment's candidates nearest first, so the same Gaussians get the same
terms but for candidates at one float distance and those before their own box entry (traverse.cuh): 0.2 %
of the paths at most, whose terms reach the order of the gradients they touch."""
import pytest
import torch

from tests.scenes import gpu_trace, gpu_trace_bwd, make_tracer, small_scene, to_torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kw", [
    (1, {}), (2, {}), (3, {}), (17, {}), (300, {}), (4000, {}), (4000, dict(kbuffer=8)), (4000, dict(block_size=64, refill_lanes=1)),
    (4000, dict(block_size=256)), (4000, dict(exact_replay=True)), (4000, dict(clamping=False)),
    (4000, dict(compensated_grads=False, warp_aggregate=False)), (60000, dict(clamping=False)),
])
def test_replay_matches_rounds_from_the_root(cuda_device, n, kw):
    s = small_scene(n=n, w=61, h=43, spp=2, max_bounces=3, scale_range=(0.02, 0.3) if n < 10000 else (0.02, 0.2))
    S = to_torch(s)
    grads = []
    for resume in (0, 1):
        tr = make_tracer(resume_rounds=resume, **kw)
        fwd = gpu_trace(tr, S)
        torch.manual_seed(5)
        g = torch.randn_like(fwd[10])
        m = torch.randn_like(fwd[7])
        _, mg, _, _, eg = gpu_trace_bwd(tr, S, fwd, g, material_grad=m)
        torch.cuda.synchronize()
        assert tr.device_status() == 0
        grads.append((mg.double(), eg.double(), tr.counters("replay")))
    (ma, ea, ca), (mb, eb, cb) = grads
    assert ca["replay"] == cb["replay"]
    assert abs(ca["replay_accepted"] - cb["replay_accepted"]) <= 0.002 * cb["replay_accepted"]
    assert float((ea - eb).norm()) <= 1e-5 * float(eb.norm())
    rows = ((ma - mb).abs() > 1e-4 * (mb.abs() + mb.norm() / max(mb.numel(), 1) ** 0.5)).any(1)
    assert float(rows.float().mean()) <= 0.02 and float((ma - mb).norm()) <= 0.02 * float(mb.norm())
