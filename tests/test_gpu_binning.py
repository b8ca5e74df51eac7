"""The binning of particles in arbitrary order (digit counts, sort tiles, fused reorder) at the edges of
its blocks and tiles: the neighbour sets are whole numbers and must equal the oracle's."""
import numpy as np
import pytest

from oracle import Oracle
from splishsplash_for_cuda_b200 import _capi
from splishsplash_for_cuda_b200.dfsph import DFSPHCUDA
from splishsplash_for_cuda_b200.scene import Configuration, Scene, box_wall
from tests._compare import neighbor_sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [1, 255, 257, 511, 512, 513, 2047, 2049, 4097])
def test_shuffled_particles(n, precision):
    r, rng = 0.025, np.random.default_rng(n)
    size = np.array((2.4, 0.5, 0.9))
    x = rng.uniform(4 * r, size - 4 * r, (n, 3)).astype(np.float32)
    walls = box_wall((0, 0, 0), tuple(size), 2 * r).astype(np.float32)
    s = Scene(config=Configuration(particleRadius=r), fluid=x, boundary=rng.permutation(walls))
    d = DFSPHCUDA(s, precision=precision, neighbor_capacity=96)
    for _ in range(2):  # the second search follows a sort of the moved (by nothing) boundary
        d.neighbors_search()
        c, l = d.neighbors()
        co, lo = Oracle(s, 64).neighbors(row=l.shape[1])
        assert d.status() & (_capi.ST_NEIGHBOR_OVERFLOW | _capi.ST_SORT_TIMEOUT | _capi.ST_ESCAPED) == 0
        assert np.array_equal(c, co)
        assert neighbor_sets(c, l) == neighbor_sets(co, lo)
        d.move_boundary_rigid(0, s.boundary.shape[0], None, (0.0, 0.0, 0.0), (0.0, 0.0, 0.0), None)


@pytest.mark.parametrize("n", [1, 513, 4097])
def test_search_applies_uploaded_velocities(n):
    """Velocities uploaded with the positions are in place after a search that re-orders the particles."""
    r, rng = 0.025, np.random.default_rng(n)
    size = np.array((2.4, 0.5, 0.9))
    x = rng.uniform(4 * r, size - 4 * r, (n, 3)).astype(np.float32)
    walls = box_wall((0, 0, 0), tuple(size), 2 * r).astype(np.float32)
    d = DFSPHCUDA(Scene(config=Configuration(particleRadius=r), fluid=x, boundary=walls), neighbor_capacity=96)
    for _ in range(3):
        x2, v2 = rng.permutation(x), rng.uniform(-1, 1, (n, 3)).astype(np.float32)
        d.update_fluid(x2, v2)
        d.neighbors_search()
        assert np.array_equal(d.velocities(), v2) and np.array_equal(d.positions(), x2)
