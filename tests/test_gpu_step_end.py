"""The pass that ends a step (position update, particles outside the domain, dt history) against the same
work in separate calls: the same bits, at the edges of its blocks."""
import numpy as np
import pytest

from splishsplash_for_cuda_b200.dfsph import DFSPHCUDA
from splishsplash_for_cuda_b200.scene import Configuration, Scene, box_wall

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 1025])
def test_step_end_matches_separate_calls(n, precision):
    r, rng = 0.025, np.random.default_rng(n)
    size = np.array((1.0, 0.8, 0.9))
    x = rng.uniform(4 * r, size - 4 * r, (n, 3)).astype(np.float32)
    v = rng.uniform(-0.2, 0.2, (n, 3)).astype(np.float32)
    v[::7] *= 4000.0  # these leave the domain in the first step
    cfg = Configuration(particleRadius=r, timeStepSize=0.001, cflMethod=1)
    s = Scene(config=cfg, fluid=x, fluid_velocity=v, boundary=box_wall((0, 0, 0), tuple(size), 2 * r).astype(np.float32))
    got = []
    for separate in (False, True):
        d = DFSPHCUDA(s, precision=precision)
        for _ in range(2):
            if separate:
                d.step_async()
                d.checkParticlesPositions(2)
            else:
                d.step()
        left = d.num_fluid()
        out = (left, [d.get_param(k) for k in ("h", "h_past", "h_future")])
        if left:
            out += (d.field("position", np.float64).tobytes(), d.field("velocity", np.float64).tobytes())
        got.append(out)
    assert got[0] == got[1]
    assert got[0][0] < n
