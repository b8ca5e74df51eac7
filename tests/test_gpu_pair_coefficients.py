"""The pair coefficients of the solver passes: list remainders (filled-up slots) against the FP64 oracle,
and the coefficients rebuilt outside the density pass."""
import numpy as np
import pytest

from oracle import Oracle
from splishsplash_for_cuda_b200.dfsph import DFSPHCUDA
from splishsplash_for_cuda_b200.scene import Configuration, Scene, box_wall, synthetic_scene
from tests._compare import assert_field

pytestmark = pytest.mark.gpu


def _sparse_block(n, seed):
    """n particles of a compressed, perforated lattice next to two walls of a box: list lengths from 0
    to about 40, with and without boundary neighbours."""
    r = 0.025
    rng = np.random.default_rng(seed)
    side = int(np.ceil((1.4 * n) ** (1.0 / 3.0))) + 1
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    x = (2.0 * r) + 1.8 * r * g[np.sort(rng.permutation(g.shape[0])[:n])] + rng.uniform(-0.1 * r, 0.1 * r, (n, 3))
    cfg = Configuration(timeStepSize=0.001, particleRadius=r)
    side_m = np.ceil((2.0 * side + 6.0)) * 2.0 * r
    return Scene(config=cfg, fluid=x.astype(np.float32), boundary=box_wall((0, 0, 0), (side_m,) * 3, 2.0 * r).astype(np.float32),
                 fluid_velocity=rng.uniform(-0.3, 0.3, (n, 3)).astype(np.float32))


# Tolerances: FP64 1e-9 as in the parity tests. FP32: 2^-24 per operation, about 16 ulp per kernel
# term, and residuals that cancel to about 1/40 of their terms over a few iterations give ~1e-4 of
# the field's scale (a velocity below a hundredth of the largest counts against that hundredth).
@pytest.mark.parametrize("precision,rtol", [(32, 1e-4), (64, 1e-9)])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 130, 257, 1025])
def test_list_remainders(n, precision, rtol):
    s = _sparse_block(n, seed=n)
    d = DFSPHCUDA(s, precision=precision)
    st = d.step()
    counts = d.field("neighbor_counts").reshape(-1, 2)
    o = Oracle(s, 64)
    ro = o.step()
    assert (st.iterations, st.iterations_v) == (ro["iterations"], ro["iterations_v"])
    if n >= 130:  # every remainder of the four-slot groups occurs
        assert set(np.unique(counts[:, 0] % 4)) == {0, 1, 2, 3} and set(np.unique(counts[:, 1] % 4)) == {0, 1, 2, 3}
    for name, floor in (("density", 1e-3), ("factor", 1e-3), ("velocity", 1e-2), ("position", 1e-3)):
        assert_field(name, d.field(name, np.float64), o.field(name), rtol, floor)


@pytest.mark.parametrize("precision", [32, 64])
def test_coefficients_rebuilt_without_a_density_pass(precision):
    """A parameter change republishes the state, after which the pressure solve forms the coefficients
    itself: the same bits as with the density pass's."""
    out = []
    for touch in (False, True):
        s = synthetic_scene(1, counts=(11, 12, 13))
        s.fluid_velocity = np.random.default_rng(3).uniform(-0.5, 0.5, s.fluid.shape).astype(np.float32)
        d = DFSPHCUDA(s, precision=precision)
        d.neighbors_search()
        d.divergence_solve()
        d.external_forces()
        d.update_time_step(0.002)
        d.update_vel()
        if touch:
            d.set_param("viscosity", d.get_param("viscosity"))
        its = d.pressure_solve()
        out.append((its, d.field("velocity", np.float64), d.field("kappa", np.float64)))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_coefficients_follow_rebuilt_lists(precision, seed):
    """Timing the neighbour build rebuilds the lists at the moved positions: the solve that follows gives
    the same bits as one that is made to form its coefficients anew."""
    out = []
    for touch in (False, True):
        s = synthetic_scene(1, counts=(11, 12, 13))
        s.fluid_velocity = np.random.default_rng(seed).uniform(-2.0, 2.0, s.fluid.shape).astype(np.float32)
        d = DFSPHCUDA(s, precision=precision)
        d.step()
        d.time_kernel("neighbor_build", 1)
        if touch:
            d.set_param("viscosity", d.get_param("viscosity"))
        d.external_forces()
        d.update_vel()
        its = d.pressure_solve()
        # bytes: alpha is scaled a second time here, and the solve may run off to NaN
        out.append((its, d.field("velocity", np.float64).tobytes(), d.field("kappa", np.float64).tobytes()))
    assert out[0] == out[1]


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 130, 257, 1025])
def test_passes_without_a_density_pass(n, precision):
    """external_forces and pressure_solve after a change that voids what the density pass left for them:
    the same bits as with it, over the list remainders."""
    out = []
    for touch in (False, True):
        s = _sparse_block(n, seed=n)
        d = DFSPHCUDA(s, precision=precision)
        void = (lambda: d.set_param("viscosity", d.get_param("viscosity"))) if touch else (lambda: None)
        d.neighbors_search()
        d.divergence_solve()
        void()
        d.external_forces()
        d.update_time_step(0.001)
        void()
        d.update_vel()
        its = d.pressure_solve()
        d.external_forces()  # with what the pressure solve has formed
        out.append((its, d.field("velocity", np.float64).tobytes(), d.field("kappa", np.float64).tobytes(),
                    d.field("acceleration", np.float64).tobytes()))
    assert out[0] == out[1]


FIELDS = ("density", "factor", "velocity", "position", "kappa", "kappa_v", "acceleration", "boundary_force")


def _state(d):
    return [d.field(name, np.float64).tobytes() for name in FIELDS]


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 130, 257, 1025])
def test_without_the_table(n, precision, learned):
    """Without the coefficient table the passes evaluate the kernel: the same bits over the list remainders,
    with forces on a moving boundary and both warm starts; and the table can come and go between steps."""
    s = _sparse_block(n, seed=n)
    out = []
    for tables in ((1, 1, 1, 1), (0, 0, 0, 0), (1, 0, 0, 1)):
        d = DFSPHCUDA(s, precision=precision)
        d.set_param("boundary_forces", 1)
        if learned:
            d.set_param("train_start", 2)
            d.set_learned_warm_start(True)
        got = []
        for k, table in enumerate(tables):
            d.set_param("pair_table", table)
            assert d.get_param("pair_table") == table
            d.move_boundary_rigid(0, s.boundary.shape[0], None, (2e-4 * k, 0.0, 0.0), (0.2, 0.0, 0.0), None)
            st = d.step()
            got += [st.iterations, st.iterations_v, _state(d)]
        out.append(got)
    assert out[0] == out[1] == out[2]


def test_a_context_that_fills_the_device_takes_no_table():
    """Lists of 0.3 of the device's memory: with as large a table less than half would stay free."""
    import torch

    s = _sparse_block(1025, seed=5)
    row = 65535
    capacity = int(0.3 * torch.cuda.mem_get_info()[1] / (4 * row))
    out = []
    for large in (False, True):
        d = DFSPHCUDA(s, **(dict(fluid_capacity=capacity, neighbor_capacity=row) if large else {}))
        assert d.get_param("pair_table") == (0 if large else 1)
        d.set_param("boundary_forces", 1)
        for _ in range(2):
            d.step()
        out.append(_state(d))
        d.close()
    assert out[0] == out[1]


def test_a_refused_table_leaves_the_context_usable():
    """A table that cannot fit is refused; the steps that follow are those of a context that never asked."""
    import torch

    from splishsplash_for_cuda_b200 import _capi

    s = _sparse_block(1025, seed=5)
    row = 65535
    capacity = int(0.55 * torch.cuda.mem_get_info()[1] / (4 * row))  # lists of 0.55 of the memory, once
    d = DFSPHCUDA(s, fluid_capacity=capacity, neighbor_capacity=row)
    small = DFSPHCUDA(s)
    for x in (d, small):
        x.set_param("boundary_forces", 1)
    with pytest.raises(_capi.DfsphError):
        d.set_param("pair_table", 1)
    assert d.get_param("pair_table") == 0
    for x in (d, small):
        x.step()
    assert _state(d) == _state(small)
    d.close()
    small.close()


def test_contexts_give_their_memory_back():
    """The device's free memory after a context with every optional array is what it was before."""
    import torch

    s = synthetic_scene(1, counts=(40, 41, 42))

    def use():
        d = DFSPHCUDA(s)
        d.set_param("pair_table", 0)
        d.set_param("boundary_forces", 1)
        d.set_learned_warm_start(True)
        d.step()
        d.set_param("pair_table", 1)
        d.step()
        d.body_wrench([0], [10], [[0.0, 0.0, 0.0]])
        d.close()

    use()  # what the first use of the library keeps (module, graphs)
    free = torch.cuda.mem_get_info()[0]
    for _ in range(5):
        use()
    assert free - torch.cuda.mem_get_info()[0] < 5 * s.n_fluid  # a leaked array has at least 4 bytes a particle
