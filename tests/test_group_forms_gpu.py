"""The neighbour kernels with 1, 2, 8 and 16 lanes per particle (SPH_GROUP_LANES)
on the same cases, bit for bit against the oracle: sizes around a warp's and a
block's particles, particles without neighbours, neighbourhoods past the masks
and the list, corners whose boundary particles pass a group's shared terms,
more repulsion candidates than are noted, batches and the closure."""
import numpy as np
import pytest

from oracle import oracle as orc
from ultraballpit_b200 import domain
from ultraballpit_b200.closure import ClosureNet
from ultraballpit_b200.kernel import (BOUNDARY_SDF, CELL_ORDER_MORTON, CELL_ORDER_ROWS, CudaBatch, CudaKernel)
from ultraballpit_b200.particles import PARTICLE_FIELDS, BoundaryParticles, ParticleArrays

from test_parity_gpu import assert_same, small_dam_break

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["1", "2", "8", "16"])
def lanes(request, monkeypatch):
    monkeypatch.setenv("SPH_GROUP_LANES", request.param)
    return int(request.param)


def first(sc, n):
    """The scenario with its first n particles."""
    p = ParticleArrays(**{f: getattr(sc.particles, f)[:n].copy() for f in PARTICLE_FIELDS})
    p.fluid_type = sc.particles.fluid_type[:n].copy()
    sc.particles = p
    return sc


def run(sc, order=CELL_ORDER_ROWS, steps=3, dt=2e-5):
    gpu = CudaKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta, cell_order=order)
    cpu = orc.OracleKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta, tier=1, threads=8, pow_mode=1)
    for _ in range(steps):
        gpu.step(dt)
        cpu.step(dt)
        assert_same(gpu.particles(), cpu.particles())
        np.testing.assert_array_equal(gpu.boundary_pressure(), cpu.boundary_pressure())
    gpu.close()


@pytest.mark.parametrize("order", [CELL_ORDER_ROWS, CELL_ORDER_MORTON])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 31, 33, 129, 1000])
def test_sizes(lanes, n, order):
    run(first(small_dam_break(), n), order)


def test_lone_particles(lanes):
    sc = first(small_dam_break(), 40)
    p = sc.particles
    p.x[:] = np.linspace(0.002, 0.078, 40, dtype=np.float32)
    p.y[:] = np.where(np.arange(40) % 2, 0.008, 0.032).astype(np.float32)
    p.z[:] = np.where(np.arange(40) % 4 < 2, 0.008, 0.032).astype(np.float32)
    run(sc)


def test_dense_block(lanes):
    # more than 128 neighbours, and neighbourhoods of more than 768 candidates
    sc = small_dam_break()
    rng = np.random.default_rng(4)
    p = sc.particles
    for a, hi in ((p.x, 0.026), (p.y, 0.036), (p.z, 0.026)):
        a[:] = rng.uniform(0.002, hi, len(p)).astype(np.float32)
    run(sc)


def test_many_boundary_particles(lanes):
    # walls 61 times as dense around a few particles in a corner: boundary terms
    # pass a group's shared terms, the list's capacity and the noted repulsion
    sc = first(small_dam_break(), 60)
    b, rng = sc.boundary, np.random.default_rng(5)
    cols = {}
    for k in ("x", "y", "z", "mass", "nx", "ny", "nz"):
        a = getattr(b, k)
        jit = rng.uniform(-0.0006, 0.0006, (60, len(a))).astype(np.float32) * np.float32(k in "xyz")
        cols[k] = np.concatenate([a] + [(a + j).astype(np.float32) for j in jit])
    sc.boundary = BoundaryParticles.from_arrays(**cols)
    p = sc.particles
    for a in (p.x, p.y, p.z):
        a[:] = rng.uniform(0.0002, 0.004, len(p)).astype(np.float32)
    run(sc)


def test_batch_equals_single_runs(lanes):
    scs = domain.batch_boxes(5, seed=3, dx=0.004, lo=200, hi=4000, draw="loguniform")
    b = CudaBatch(scs)
    b.step_auto(4)
    for q, sc in enumerate(scs):
        k = CudaKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta)
        k.step_auto(4)
        assert_same(b.instance(q), k.particles())
        k.close()
    b.close()


@pytest.mark.parametrize("mode", [1, 2])
def test_closure_and_sdf_walls_equal_the_thread_form(lanes, mode, monkeypatch):
    sc = domain.tank_with_sphere(0.004, domain_max=(0.048, 0.048, 0.06), center=(0.024, 0.024, 0.02), radius=0.01,
                                 fill_height=0.04, hydrostatic=True, geometry="lattice")
    out = []
    for form in (str(lanes), "1"):
        monkeypatch.setenv("SPH_GROUP_LANES", form)
        for kw in ({}, dict(boundary_mode=BOUNDARY_SDF, sdf=sc.obstacle_sdf)):
            k = CudaKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta, **kw)
            if not kw:
                k.set_feature_sdf(sc.sdf)
            k.set_closure(mode, ClosureNet(seed=2).params() if mode == 2 else None)
            k.step_auto(3)
            ids, feat, rho = k.closure_samples()
            o = np.argsort(ids)
            out.append((k.particles(), ids[o], feat[o], rho[o]))
            k.close()
    for a, b in zip(out[:2], out[2:]):
        assert_same(a[0], b[0])
        for x, y in zip(a[1:], b[1:]):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("n", [1, 3, 15, 16, 17, 63, 115])
def test_closure_at_a_tile_s_and_a_block_s_edges(lanes, n, monkeypatch):
    """A tile of the network holds 16 particles; a block of the group forms' 8
    or 16 shares one, whatever part of them is there and near the wall."""
    out = []
    for form in (str(lanes), "1"):
        monkeypatch.setenv("SPH_GROUP_LANES", form)
        sc = first(domain.tank_with_sphere(0.004, domain_max=(0.02, 0.02, 0.03), center=(0.01, 0.01, 0.008),
                                           radius=0.005, fill_height=0.018, geometry="lattice"), n)
        k = CudaKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta)
        k.set_feature_sdf(sc.sdf)
        k.set_closure(2, ClosureNet(seed=4).params())
        k.step_auto(2)
        ids, feat, rho = k.closure_samples()
        o = np.argsort(ids)
        out.append((k.particles(), ids[o], feat[o], rho[o]))
        k.close()
    assert_same(out[0][0], out[1][0])
    for x, y in zip(out[0][1:], out[1][1:]):
        np.testing.assert_array_equal(x, y)
