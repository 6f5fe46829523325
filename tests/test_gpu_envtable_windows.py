"""Device-built alias tables around the sizes of the pairing's windows (1280 cells of either list) and with lists
of extreme length. What a table samples (a cell's own probability plus what aliases to it) has to be the
distribution its pdf states: pdf times the cell's solid angle, in 64 bits. The table holds float32, so a cell may be off
by one rounding (2^-24) of the pdf, of its own probability and of each that aliases to it, with a factor of two, and by the
float32 rounding of the cell weights and their total."""
import numpy as np
import pytest
import torch

from ptir_b200 import envmap

pytestmark = pytest.mark.gpu


def _cube(fs, kind):
    rng = np.random.default_rng(fs)
    e = np.ones((6 * fs, fs, 4), np.float32)
    if kind == "lognormal":
        e[..., :3] = rng.lognormal(0.0, 1.0, (6 * fs, fs, 3))
    elif kind == "one bright":  # one large cell takes every small one
        e[..., :3] = 1e-3
        e[fs, 1 % fs, :3] = 1e4
    elif kind == "one dark":  # one small cell far below the rest, which lie around 1
        e[2 * fs, 0, :3] = 0.0
    elif kind == "halves":  # long runs of either kind
        e[: 3 * fs, :, :3] = 3.0
    return torch.from_numpy(e)


def _solid(fs):
    e = np.linspace(-1.0, 1.0, fs + 1)
    area = lambda u, v: np.arctan2(u * v, np.sqrt(u * u + v * v + 1.0))  # noqa: E731
    u0, u1, v0, v1 = e[None, :-1], e[None, 1:], e[:-1, None], e[1:, None]
    return np.tile(area(u1, v1) - area(u0, v1) - area(u1, v0) + area(u0, v0), (6, 1)).reshape(-1)


@pytest.mark.parametrize("kind", ["lognormal", "one bright", "one dark", "halves"])
@pytest.mark.parametrize("fs", [1, 2, 14, 15, 20, 21, 29, 40])
def test_table_samples_its_pdf(cuda_device, fs, kind):
    prob, alias, pdf = envmap.build_device(_cube(fs, kind).to(cuda_device)).cpu().numpy().astype(np.float64).reshape(3, -1)
    n = prob.size
    target = alias.astype(np.int64)
    assert np.all((prob >= 0.0) & (prob <= 1.0)) and np.all((target >= 0) & (target < n))
    mass = prob.copy()
    np.add.at(mass, target, 1.0 - prob)
    sources = np.bincount(target, minlength=n)
    want = pdf * _solid(fs) * n
    eps = 2.0 ** -24
    assert np.all(np.abs(mass - want) <= 2.0 * eps * (2.0 + sources) + 8.0 * eps * want + 1e-12 * n)
