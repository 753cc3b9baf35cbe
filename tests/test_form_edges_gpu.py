"""Edges of the forms that the neighbour kernels take by size (SPH_GROUP_LANES
sets the lanes per particle): instances without particles, particles in
neighbourhoods past the scan's masks, coefficients and densities outside the
ordinary, and the paths taken only by large grids or without a boundary list."""
import numpy as np
import pytest

from oracle import oracle as orc
from ultraballpit_b200 import domain
from ultraballpit_b200.closure import ClosureNet
from ultraballpit_b200.kernel import CELL_ORDER_LINEAR, CELL_ORDER_ROWS, CudaBatch, CudaKernel
from ultraballpit_b200.particles import BoundaryParticles, ParticleArrays

from test_group_forms_gpu import first
from test_parity_gpu import assert_same, small_dam_break

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("empty", [0, 1, 2])
@pytest.mark.parametrize("lanes", ["1", "8", "16"])
def test_timestep_of_an_instance_without_particles(lanes, empty, monkeypatch):
    monkeypatch.setenv("SPH_GROUP_LANES", lanes)
    scs = [first(small_dam_break(seed), 0 if q == empty else 300) for q, seed in enumerate((3, 4, 5))]
    b = CudaBatch(scs)
    for _ in range(2):
        b.step_each([1e-5, 2e-5, 3e-5])
    want = b.timesteps()
    sc = scs[empty]
    f = np.float32
    assert want[empty] == f(sc.cfl_number) * f(sc.h) / f(sc.speed_of_sound)  # nothing moves: the signal speed's
    dt = b.step_auto(1)
    assert f(dt) == want[0]
    b.close()


@pytest.mark.parametrize("lanes", ["1", "2", "8", "16"])
def test_close_pair_in_a_crowded_neighbourhood(lanes, monkeypatch):
    """Three particles 1e-13 and 3e-12 apart, alone in their support, with 900 more beyond it in the cells around:
    too many candidates for the scan's masks, and a distance below 1e-12, where the kernel's gradient is zero."""
    monkeypatch.setenv("SPH_GROUP_LANES", lanes)
    h = np.float32(1.3 * 0.004)
    cell = np.float32(2.0) * h
    rng = np.random.default_rng(1)
    x, y, z = (rng.uniform(lo, 0.0205, 903).astype(np.float32) for lo in (0.015, 0.0, 0.0))
    x[:3], y[:3], z[:3] = (0.0, 1e-13, 0.0), (0.0, 0.0, 3e-12), 0.0
    p = ParticleArrays.from_positions(x, y, z, 6.4e-5)
    p.mass[:3] *= 4  # their density above the rest density, so that they press on one another
    p.mass[3:] *= np.float32(0.05)
    p.vx[0], p.vy[2] = 0.5, -0.5
    none = BoundaryParticles.from_arrays(*[np.zeros(0, np.float32)] * 7)
    args = (p, none, float(h), (0.0, 0.0, -9.81), 20.0, 0.25, 0.0, (float(-2 * cell),) * 3, (float(8 * cell),) * 3)
    gpu = CudaKernel(*args)
    cpu = orc.OracleKernel(*args, tier=1, threads=8, pow_mode=1)
    assert [len(gpu.neighbors(q)) for q in range(3)] == [2, 2, 2]
    for _ in range(3):
        gpu.step(1e-7)
        cpu.step(1e-7)
        assert_same(gpu.particles(), cpu.particles())
    gpu.close()


def forces_us(k):
    return min(k.step_profiled(2e-5)["forces_us"] for _ in range(12))


def alone(sc, q, mass):
    """Particles q of the scenario in the middle of its empty part, with the given mass."""
    p = sc.particles
    p.mass[q], p.x[q], p.y[q], p.z[q] = mass, 0.25, 0.1, 0.05


def passing(sc):  # two particles in one place, denser together than 2^30, that part at once
    alone(sc, [4, 5], 200.0)
    sc.particles.vx[4], sc.particles.vx[5] = -700.0, 700.0


def thin(sc):  # a particle by itself whose density is far below any fluid's
    alone(sc, [4], 1e-15)


def light(sc):  # masses of a very fine discretisation
    alone(sc, [4], 1e-20)


@pytest.mark.parametrize("lanes", ["1", "8"])
@pytest.mark.parametrize("change", [passing, thin, light])
def test_an_odd_particle_does_not_slow_the_rest(change, lanes, monkeypatch):
    """The sums of all particles leave their lists for a grid search (5 to 9 times the forces' time) while a density
    or mass of the simulation is outside what the quick quotients allow, and only then."""
    monkeypatch.setenv("SPH_GROUP_LANES", lanes)
    times = []
    for f in (None, change):
        sc = domain.dam_break(0.004, seed=3, block=(0.1, 0.2, 0.1), domain_max=(0.4, 0.2, 0.1), with_sdf=False)
        if f:
            f(sc)
        gpu = CudaKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta)
        if f:
            cpu = orc.OracleKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta, tier=1, threads=8, pow_mode=1)
            for _ in range(3):
                gpu.step(2e-5)
                cpu.step(2e-5)
                assert_same(gpu.particles(), cpu.particles())
        times.append(forces_us(gpu))
        gpu.close()
    assert times[1] < 2.0 * times[0], times


@pytest.mark.parametrize("lanes", ["1", "8"])
@pytest.mark.parametrize("coef", [(-0.5, 2.0), (0.5, -2.0), (-0.5, -2.0), (-1e-25, 1.0), (1e-25, -1.0)])
def test_negative_viscous_coefficients(coef, lanes, monkeypatch):
    """Velocities over 34 decades: viscous dividends whose two parts cancel or underflow, some to nothing."""
    monkeypatch.setenv("SPH_GROUP_LANES", lanes)
    sc = small_dam_break()
    p, rng = sc.particles, np.random.default_rng(9)
    for a in (p.vx, p.vy, p.vz):
        a[:] = (rng.uniform(-1, 1, len(p)) * 10.0 ** rng.uniform(-34, 0, len(p))).astype(np.float32)
    gpu = CudaKernel(*sc.kernel_args(), alpha=coef[0], beta=coef[1])
    cpu = orc.OracleKernel(*sc.kernel_args(), alpha=coef[0], beta=coef[1], tier=1, threads=8, pow_mode=1)
    for _ in range(3):
        gpu.step(2e-5)
        cpu.step(2e-5)
        assert_same(gpu.particles(), cpu.particles())
    gpu.close()


@pytest.mark.parametrize("lanes", ["1", "8"])
def test_negative_viscous_coefficients_keep_the_lists(lanes, monkeypatch):
    monkeypatch.setenv("SPH_GROUP_LANES", lanes)
    times = []
    for alpha in (0.5, -0.5):
        sc = domain.dam_break(0.004, seed=3, block=(0.1, 0.2, 0.1), domain_max=(0.4, 0.2, 0.1), with_sdf=False)
        gpu = CudaKernel(*sc.kernel_args(), alpha=alpha, beta=sc.beta)
        times.append(forces_us(gpu))
        gpu.close()
    assert times[1] < 2.0 * times[0], times


def test_tuned_shapes_belong_to_the_form(monkeypatch):
    """The forms change inside a bin of the size histogram: shapes tuned for one are not handed to another."""
    sc = first(small_dam_break(), 777)
    best = {}
    for lanes in ("8", "1", "8", "1"):
        monkeypatch.setenv("SPH_GROUP_LANES", lanes)
        k = CudaKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta)
        before = k.particles()
        got = k.autotune(2)
        k._cache = None
        cached = np.array_equal(before.z, k.particles().z)
        assert cached == (lanes in best)  # a cache hit runs no step
        assert best.setdefault(lanes, got) == got == k.launch()
        assert lanes == "1" or set(got.values()) == {128}  # nothing to choose
        k.close()


def test_closure_modes_of_a_wide_block(monkeypatch):
    """The density kernel of each closure mode with 512 threads a block, whose shared memory passes the default limit:
    each mode's kernel is allowed it when the mode is set."""
    monkeypatch.setenv("SPH_GROUP_LANES", "1")
    sc = domain.tank_with_sphere(0.004, domain_max=(0.048, 0.048, 0.06), center=(0.024, 0.024, 0.02), radius=0.01,
                                 fill_height=0.04, hydrostatic=True, geometry="lattice")
    out = []
    for threads in (128, 512):
        k = CudaKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta)
        k.set_launch(128, threads, 128)
        k.set_feature_sdf(sc.sdf)
        for mode in (0, 2, 1, 0):
            k.set_closure(mode, ClosureNet(seed=2).params() if mode == 2 else None)
            k.step_auto(2)
        out.append(k.particles())
        k.close()
    assert_same(*out)


@pytest.mark.parametrize("lanes", ["1", "2", "8", "16"])
def test_boundary_pressure_without_lists(lanes, monkeypatch):
    """The search that stands in where the boundary particles' lists have no memory."""
    monkeypatch.setenv("SPH_GROUP_LANES", lanes)
    monkeypatch.setenv("SPH_WALL_LISTS", "0")
    sc = small_dam_break()
    gpu = CudaKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta)
    cpu = orc.OracleKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta, tier=1, threads=8, pow_mode=1)
    for _ in range(3):
        gpu.step(2e-5)
        cpu.step(2e-5)
        assert_same(gpu.particles(), cpu.particles())
        np.testing.assert_array_equal(gpu.boundary_pressure(), cpu.boundary_pressure())
    gpu.close()


def test_boundary_pressure_of_a_batch_without_lists(monkeypatch):
    scs = domain.batch_boxes(3, seed=5, dx=0.004, lo=200, hi=2000, draw="loguniform")
    out = []
    for lists in ("1", "0"):
        monkeypatch.setenv("SPH_WALL_LISTS", lists)
        b = CudaBatch(scs)
        b.step_auto(4)
        out.append((b.particles(), b.boundary_pressure()))
        b.close()
    assert_same(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    assert out[0][1].any()


# cells of the grid: one scan kernel up to 16,384, two up to 2,097,152, three above
@pytest.mark.parametrize("dims", [(32, 32, 16), (41, 40, 10), (128, 128, 128), (129, 128, 128), (300, 90, 90)])
@pytest.mark.parametrize("order", [CELL_ORDER_ROWS, CELL_ORDER_LINEAR])
def test_grids_of_many_cells(dims, order):
    h = np.float32(1.3 * 0.004)
    cell = np.float32(2.0) * h
    hi = tuple(float(np.float32((d - 0.5) * cell)) for d in dims)
    rng = np.random.default_rng(3)
    # clumps of neighbours all over the grid, and particles in its first and last cells
    centre = rng.uniform(0.1, 0.9, (60, 3)) * hi
    x = (centre[:, None, :] + rng.uniform(-0.4, 0.4, (60, 10, 3)) * cell).reshape(-1, 3)
    x[0], x[1] = 0.1 * cell, np.array(hi) - 0.1 * cell
    p = ParticleArrays.from_positions(*x.T.astype(np.float32), 6.4e-5)
    none = BoundaryParticles.from_arrays(*[np.zeros(0, np.float32)] * 7)
    args = (p, none, float(h), (0.0, 0.0, -9.81), 20.0, 0.25, 0.0, (0.0, 0.0, 0.0), hi)
    gpu = CudaKernel(*args, cell_order=order)
    g = gpu.read_grid()
    o = orc.grid_build(p.x, p.y, p.z, cell, args[7], args[8])
    assert tuple(g["dims"]) == o["dims"] == dims
    np.testing.assert_array_equal(g["cell_count"], o["counts"])
    if order == CELL_ORDER_LINEAR:
        np.testing.assert_array_equal(g["cell_start"], o["offsets"])
        np.testing.assert_array_equal(g["slot_id"], o["sorted"])
    cpu = orc.OracleKernel(*args, tier=1, threads=8, pow_mode=1)
    for _ in range(3):
        gpu.step(2e-5)
        cpu.step(2e-5)
        assert_same(gpu.particles(), cpu.particles())
    gpu.close()
