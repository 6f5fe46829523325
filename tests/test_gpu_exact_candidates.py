"""``exact_candidates``: every traversal, the shadow rays' and the replay's among them, returns the K nearest
candidates whatever its order. So the four-lane kernels of a small launch find as many candidates, in as many calls, as
the megakernel, and a replay scatters to the same Gaussians whether its rounds resume or start at the root.
Elongated Gaussians with a clamped support, of which some rays graze a box and meet the closest approach before it. Counts
are equal. Of gradients the sum over the Gaussians is compared: resumed rounds come to candidates at one and the same
float distance in another order, which moves weight between their rows and leaves its sum; float32 rounding of the
rows stays below 1e-5 of the sum of their sizes."""
import pytest
import torch

from tests.scenes import gpu_trace, gpu_trace_bwd, make_tracer, small_scene, to_torch

pytestmark = pytest.mark.gpu

COUNTS = ("segments", "trace_calls", "candidates", "accepted")


def _scene(n, seed):
    big = n > 5000
    return to_torch(small_scene(n=n, w=96 if big else 64, h=80 if big else 48, spp=2, max_bounces=4, seed=seed,
                                scale_range=(0.002, 0.3) if big else (0.005, 0.5)))


@pytest.mark.parametrize("n,seed", [(3000, 1), (3000, 2), (10000, 1)])
def test_shadow_rays_find_what_the_megakernel_finds(cuda_device, n, seed):
    S = _scene(n, seed)
    got = []
    for schedule in ("wavefront", "megakernel"):
        tr = make_tracer(exact_candidates=True, schedule=schedule)
        gpu_trace(tr, S)
        got.append([tr.counters()[k] for k in COUNTS])
        assert tr.device_status() == 0
    assert got[0] == got[1]


@pytest.mark.parametrize("n,seed", [(3000, 1), (10000, 1), (10000, 2)])
def test_replay_does_not_depend_on_its_rounds(cuda_device, n, seed):
    S = _scene(n, seed)
    got = []
    for resume in (0, 1):
        tr = make_tracer(exact_candidates=True, resume_rounds=resume)
        fwd = gpu_trace(tr, S)
        torch.manual_seed(1)
        _, mg, _, _, _ = gpu_trace_bwd(tr, S, fwd, torch.randn_like(fwd[10]), material_grad=torch.randn_like(fwd[7]))
        c = tr.counters("replay")
        got.append((c["replay"], c["replay_accepted"], mg))
        assert tr.device_status() == 0
    (ja, aa, ma), (jb, ab, mb) = got
    assert (ja, aa) == (jb, ab)
    ma, mb = ma.double(), mb.double()
    assert bool(((ma.sum(0) - mb.sum(0)).abs() <= 1e-5 * mb.abs().sum(0)).all())
