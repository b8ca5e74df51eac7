"""The binning of particles in arbitrary order (digit counts, sort tiles, fused reorder) at the edges of
its blocks and tiles: the neighbour sets are whole numbers and must equal the oracle's."""
import time

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


def test_few_particles_in_a_large_domain():
    """The binning also clears the cell table, which is far larger than a small set: not in a few blocks.
    Bounds: 8 bytes a cell at a tenth of 6.4 TB/s, and 0.2 ms (1 ms for a host call) for everything else."""
    r, cells, rng = 0.025, 400, np.random.default_rng(7)
    x = rng.uniform(1.0, 1.5, (1000, 3)).astype(np.float32)
    b = rng.uniform(1.0, 2.0, (500, 3)).astype(np.float32)
    s = Scene(config=Configuration(particleRadius=r), fluid=x, boundary=b)
    small, large = (DFSPHCUDA(s, neighbor_capacity=512, grid_box=(0, 0, 0) + (side,) * 3) for side in (2.5, cells * 4 * r))
    clear = 8.0 * cells ** 3 / 0.64e12
    for _ in range(2):
        assert min(large.time_kernel("sort_reorder", 1) * 1e-3 for _ in range(5)) < clear + 0.2e-3
        took = []
        for d in (small, large):
            d.neighbors_search()
        assert small.status() == large.status() == 0
        assert np.array_equal(small.field("neighbor_counts"), large.field("neighbor_counts"))
        for _ in range(5):
            t = time.perf_counter()
            large.move_boundary(b)
            large.synchronize()
            took.append(time.perf_counter() - t)
        assert min(took) < clear + 1e-3
        small.move_boundary(b)
    small.close()
    large.close()


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [1, 513, 4097])
def test_fluid_and_boundary_binnings_alternate(n, precision):
    """Both sets are sorted with the same buffers: searches between re-binnings of the boundary at its
    unchanged positions (a part of it moved by nothing, and all of it uploaded again) find the same sets."""
    r, rng = 0.025, np.random.default_rng(n)
    size = np.array((2.4, 0.5, 0.9))
    x = rng.uniform(4 * r, size - 4 * r, (n, 3)).astype(np.float32)
    walls = rng.permutation(box_wall((0, 0, 0), tuple(size), 2 * r).astype(np.float32))
    s = Scene(config=Configuration(particleRadius=r), fluid=x, boundary=walls)
    d = DFSPHCUDA(s, precision=precision, neighbor_capacity=96)
    co, lo = Oracle(s, 64).neighbors(row=96)
    part = lambda: d.move_boundary_rigid(0, walls.shape[0] - 1, None, (0.0, 0.0, 0.0), (0.0, 0.0, 0.0), None)
    for bins in ((), (part,), (lambda: d.move_boundary(walls),), (part, part, lambda: d.move_boundary(walls)), ()):
        for again in bins:
            again()
        d.neighbors_search()
        c, l = d.neighbors(96)
        assert d.status() & (_capi.ST_NEIGHBOR_OVERFLOW | _capi.ST_SORT_TIMEOUT | _capi.ST_ESCAPED) == 0
        assert np.array_equal(c, co)
        assert neighbor_sets(c, l) == neighbor_sets(co, lo)


def test_lists_read_before_and_after_a_search():
    """The lists come in groups of the longest one: none before the first search, a far longer one after a
    part of the fluid has been pressed together."""
    r, rng = 0.025, np.random.default_rng(3)
    x = rng.uniform(0.06, 0.94, (1500, 3)).astype(np.float32)
    walls = box_wall((0, 0, 0), (1.0, 1.0, 1.0), 2 * r).astype(np.float32)
    s = Scene(config=Configuration(particleRadius=r), fluid=x, boundary=walls)
    d = DFSPHCUDA(s)
    c, l = d.neighbors()
    assert not c.any()
    for scale in (1.0, 0.5):  # lists of up to 19 and 87, the oracle holds 96
        s.fluid = (0.5 + scale * (x - 0.5)).astype(np.float32)
        d.update_fluid(s.fluid)
        d.neighbors_search()
        c, l = d.neighbors()
        co, lo = Oracle(s, 64).neighbors(row=l.shape[1])
        assert np.array_equal(c, co) and neighbor_sets(c, l) == neighbor_sets(co, lo)
