"""Whole paths and their adjoint above and below 131,072 rays a launch: eight views of 120,000 paths traced alone (four
lanes a ray in every stage) and together (one lane a ray, sorted queues). A path's draws depend on its pixel and
frame, not on the launch. Without density clamping, launches differ in the order of candidates at one and the
same float distance, which up to 0.5 % of segments have; a path here has up to four (primary, shadow ray, two
bounces), so 2 % of the paths may differ. The environment gradients are the views' summed: 2e-3 of their norm, as between
the schedules. The material gradient is compared Gaussian by Gaussian: a launch of more rays than threads seeds a call from
whichever segment the lane had before, which in one path of 100,000 changes whether a grazing candidate is kept, and one
path of large radiance can hold more than 2e-3 of the norm. Some ten paths of these 960,000, of up to 100 Gaussians each,
reach half of the 2,000 at most; for the other half eight float32 sums, each compensated to an ulp of its size, leave less
than 1e-5 of the row."""
import pytest
import torch

from ptir_b200 import synthetic
from tests.scenes import make_tracer, small_scene, to_torch
from tests.test_gpu_views import _scene_args, _tail

pytestmark = pytest.mark.gpu

LINE, VIEWS, W, H = 131_072, 8, 400, 300


def _trace(tr, S, views, ori, dirs, grads):
    fwd = [t.clone() for t in tr.trace_views(views, ori, dirs, *_scene_args(S), *_tail(S))]
    ctr = {k: tr.counters(k)["segments"] for k in ("intersect", "shadow")}
    z = torch.zeros_like
    bwd = tr.trace_bwd_views(views, ori, dirs, *fwd[:8], fwd[10], fwd[11], *_scene_args(S), *[z(t) for t in fwd[:7]],
                             grads[1], grads[0], z(fwd[11]), *_tail(S))
    ctr["replay"] = tr.counters("replay")["replay"]
    torch.cuda.synchronize()
    assert tr.device_status() == 0
    return fwd, bwd[1].double(), bwd[4].double(), ctr


@pytest.mark.parametrize("kw", [{}, dict(kbuffer=8), dict(shadow_kbuffer=8), dict(exact_candidates=True),
                                dict(sort_rays=False), dict(resume_rounds=1), dict(storage="bf16")])
def test_views_together_trace_as_alone(cuda_device, kw):
    S = to_torch(small_scene(n=2000, max_bounces=3, scale_range=(0.05, 0.3)))
    tr = make_tracer(clamping=False, **kw)
    tr.build_bvh(S["build_pos"], S["build_rot"], S["build_scl"], S["build_dns"], True, True)
    eyes = synthetic.camera_positions(VIEWS, seed=2)
    views = [(k, S["ray_to_world"], 1, H, W) for k in range(VIEWS)]
    rays = [[t.to(cuda_device).reshape(-1, 3) for t in synthetic.view_rays(W, H, 1, e)] for e in eyes]
    n = W * H
    g = torch.Generator(device="cuda").manual_seed(1)
    grads = [torch.randn((VIEWS * n, c), generator=g, device="cuda") for c in (3, 5)]
    ori, dirs = (torch.cat([r[k] for r in rays]) for k in (0, 1))
    fwd, mg, eg, ctr = _trace(tr, S, views, ori, dirs, grads)
    # of the two bounce and the three replay launches at least one is above the line
    assert ctr["shadow"] > LINE and ctr["intersect"] - VIEWS * n > 2 * LINE and ctr["replay"] > 3 * LINE, ctr
    differ, mg_sum, eg_sum, seen = 0, torch.zeros_like(mg), torch.zeros_like(eg), torch.zeros_like(fwd[9])
    for k in range(VIEWS):
        part = slice(k * n, (k + 1) * n)
        f, m, e, _ = _trace(tr, S, views[k:k + 1], *rays[k], [t[part] for t in grads])
        same = torch.ones(n, dtype=torch.bool, device=cuda_device)
        for i, (a, b) in enumerate(zip(f, fwd)):
            if i != 9:
                same &= (a.reshape(n, -1) == b[part].reshape(n, -1)).all(1)
        differ += int((~same).sum())
        mg_sum, eg_sum, seen = mg_sum + m, eg_sum + e, torch.maximum(seen, f[9])
    assert differ <= 0.02 * VIEWS * n, differ
    assert int((seen != fwd[9]).sum()) <= 0.002 * seen.numel()
    assert float((eg_sum - eg).norm()) <= 2e-3 * float(eg.norm())
    rows = mg.norm(dim=1)
    assert float(((mg_sum - mg).norm(dim=1)[rows > 0] / rows[rows > 0]).median()) <= 1e-5
