"""Device-built alias tables around the sizes of the pairing's windows (1280 cells of either list) and with lists
of extreme length, against the host table: tolerances of test_gpu_envtable.py (the device's weights
differ from the host's in the last bits, which may end the pairing one cell sooner or later)."""
import numpy as np
import pytest
import torch

from ptir_b200 import envmap
from tests.test_gpu_envtable import _mass

pytestmark = pytest.mark.gpu


def _cube(fs, kind):
    rng = np.random.default_rng(fs)
    e = np.ones((6 * fs, fs, 4), np.float32)
    if kind == "lognormal":
        e[..., :3] = rng.lognormal(0.0, 1.0, (6 * fs, fs, 3))
    elif kind == "one bright":  # one large cell takes every small one
        e[..., :3] = 1e-3
        e[fs, 1, :3] = 1e4
    elif kind == "one dark":  # one small cell far below the rest, which lie around 1
        e[2 * fs, 0, :3] = 0.0
    elif kind == "halves":  # long runs of either kind
        e[: 3 * fs, :, :3] = 3.0
    return torch.from_numpy(e)


@pytest.mark.parametrize("kind", ["lognormal", "one bright", "one dark", "halves"])
@pytest.mark.parametrize("fs", [1, 2, 14, 15, 20, 21, 29, 40])
def test_table_at_window_sizes(cuda_device, fs, kind):
    env = _cube(fs, kind)
    host = envmap.pack(envmap.build(env, cube=True)).numpy()
    dev = envmap.build_device(env.to(cuda_device)).cpu().numpy()
    np.testing.assert_allclose(dev[2], host[2], rtol=1e-5, atol=1e-12)
    m_dev, m_host = (_mass(t[0].reshape(-1), t[1].reshape(-1)) for t in (dev, host))
    np.testing.assert_allclose(m_dev, m_host, rtol=1e-5, atol=1e-10)
