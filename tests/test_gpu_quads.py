"""The two forms of the intersection stage: four lanes a ray in small launches, one lane a ray above 131,072
rays. The same primary rays are traced in one launch of 180,000 and in slices of it that stay below the line.
Without density clamping a primary ray's outputs do not depend on the launch: only the order of
candidates at one and the same float distance may, which up to 0.5 % of rays have (distances of order 1 in
steps of 2^-23, some fifty candidates a ray)."""
import pytest
import torch

from tests.scenes import gpu_trace, make_tracer, small_scene, to_torch

pytestmark = pytest.mark.gpu


def _trace(S, ori, dirs, **kw):
    tr = make_tracer(clamping=False, mis=False, **kw)
    out = gpu_trace(tr, dict(S, ray_ori=ori, ray_dir=dirs))
    torch.cuda.synchronize()
    assert tr.device_status() == 0
    return [t for k, t in enumerate(out) if k not in (2, 9)] + [out[2][..., :1]], out[9]


@pytest.mark.parametrize("n,kw", [
    (0, {}), (1, {}), (2, {}), (5, {}), (17, {}), (3000, {}), (3000, dict(kbuffer=8)), (3000, dict(exact_candidates=True)),
    (3000, dict(storage="bf16")), (3000, dict(block_size=64, refill_lanes=5)), (3000, dict(block_size=256, refill_lanes=1)),
])
def test_small_launches_trace_as_large_ones(cuda_device, n, kw):
    s = small_scene(n=max(n, 1), w=450, h=400, spp=1, max_bounces=1, scale_range=(0.02, 0.2))
    S = to_torch(s)
    if n == 0:
        S = {k: (v[:0] if k.startswith("build_") or k in ("density", "material", "sph", "shading_normal") else v)
             for k, v in S.items()}
    ori, dirs = S["ray_ori"], S["ray_dir"]
    whole, vis = _trace(S, ori, dirs, **kw)
    seen = torch.zeros_like(vis)
    rows = same = 0
    for a, b in ((0, 1), (1, 8), (8, 150), (150, 400)):
        part, v = _trace(S, ori[:, a:b].contiguous(), dirs[:, a:b].contiguous(), **kw)
        seen = torch.maximum(seen, v)
        eq = torch.ones(((b - a) * 450,), dtype=torch.bool, device=cuda_device)
        for x, y in zip(part, whole):
            eq &= (x.reshape(eq.numel(), -1) == y[:, a:b].reshape(eq.numel(), -1)).all(1)
        rows += eq.numel()
        same += int(eq.sum())
    assert same >= (rows if n <= 5 else 0.995 * rows), (same, rows)
    assert int((seen != vis).sum()) <= (0 if n <= 17 else 3)


def test_coincident_gaussians(cuda_device):
    """Every candidate of a ray at one distance: the k-buffer takes the first sixteen it meets."""
    s = small_scene(n=200, w=450, h=400, spp=1, max_bounces=1)
    for k in ("build_pos", "build_rot", "build_scl", "build_dns", "density", "material", "sph", "shading_normal"):
        s[k][:] = s[k][:1]
    for k in ("build_scl", "density"):
        s[k][:, (8 if k == "density" else 0):(11 if k == "density" else 3)] = 0.4
    S = to_torch(s)
    whole, _ = _trace(S, S["ray_ori"], S["ray_dir"])
    part, _ = _trace(S, S["ray_ori"][:, 100:300].contiguous(), S["ray_dir"][:, 100:300].contiguous())
    for x, y in zip(part, whole):
        assert torch.equal(x, y[:, 100:300])
