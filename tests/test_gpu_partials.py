"""The last block's walk over the block partials (CFL maximum, residual sums) at the edges of its batches:
lattices of about 1, 8 and 9 rounds of its 256 threads."""
import numpy as np
import pytest

from splishsplash_for_cuda_b200.dfsph import DFSPHCUDA
from splishsplash_for_cuda_b200.scene import Configuration, Scene, box_wall

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [1, 255, 256, 257, 2047, 2048, 2049])
def test_maximum_and_mean_reach_every_block(blocks):
    """Particles too far apart to interact, one of them fast: the CFL step follows the fastest one wherever
    its block stands, and every residual is zero."""
    n = 256 * (blocks - 1) + 1  # the last block holds one particle
    r = 0.01
    side = int(np.ceil(n ** (1.0 / 3.0)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)[:n]
    x = ((g + 1.0) * 5.0 * r).astype(np.float32)
    walls = box_wall((0, 0, 0), ((side + 2) * 5.0 * r,) * 3, 20 * r).astype(np.float32)
    cfg = Configuration(particleRadius=r, timeStepSize=1e-4, cflMethod=1, cflFactor=0.5, cflMaxTimeStepSize=1.0,
                        viscosity=0.0, gravitation=(0.0, 0.0, 0.0))
    for fast in sorted({0, n // 2, n - 1}):
        v = np.zeros((n, 3), np.float32)
        v[fast] = (3.0, 0.0, 0.0)
        d = DFSPHCUDA(Scene(config=cfg, fluid=x, fluid_velocity=v, boundary=walls))
        st = d.step()
        assert st.density_error == 0.0 and st.divergence_error == 0.0
        assert abs(st.h_future - 0.5 * 0.4 * 2.0 * r / 3.0) <= 1e-12  # vmax^2 = 9 exactly in FP32
        d.close()


@pytest.mark.parametrize("blocks", [1, 2, 255, 256, 257, 2047, 2048, 2049, 2305])
def test_mean_of_nonzero_residuals(blocks):
    """A compressed lattice with disorder, where every block's partial is another number: the mean residual
    that ends the pressure loop is the FP64 mean of the particles' residuals. A block left out or taken twice
    shows as 1 / blocks; FP64 sums of some 40 levels differ from the host's by 1e-14."""
    n = 256 * (blocks - 1) + 1
    r, rng = 0.01, np.random.default_rng(blocks)
    side = int(np.ceil(n ** (1.0 / 3.0)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)[:n]
    x = ((g + 3.0) * 1.7 * r + rng.uniform(-0.1 * r, 0.1 * r, (n, 3))).astype(np.float32)
    walls = box_wall((0, 0, 0), ((side + 6) * 1.7 * r,) * 3, 20 * r).astype(np.float32)
    cfg = Configuration(particleRadius=r, timeStepSize=1e-4, maxIterations=3, maxIterationsV=1)
    d = DFSPHCUDA(Scene(config=cfg, fluid=x, boundary=walls), neighbor_capacity=128)
    d.set_param("remove_escaped", 0)  # the walls' last plane can lie before the lattice's
    st = d.step()
    residual = d.field("density_adv").astype(np.float64)
    assert d.num_fluid() == n and (n == 1 or residual.max() > 0)
    assert abs(st.density_error - residual.mean()) <= 1e-13 * residual.mean()
    d.close()
