"""The pair sums' square root, reciprocal and quotient (sph::sqrt_rn, rcp_rn,
div_rn) against CUDA's IEEE operations, and the particles whose operands leave
the range where those are exact: they are recomputed with the general
operations, so every state below must still equal the oracle bit for bit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle as orc
from ultraballpit_b200 import domain
from ultraballpit_b200.kernel import CELL_ORDER_MORTON, CELL_ORDER_ROWS, CudaKernel

from test_parity_gpu import assert_same, small_dam_break

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def arith(tmp_path_factory):
    out = tmp_path_factory.mktemp("arith") / "libarith.so"
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--fmad=false",
                    "-prec-div=true", "-prec-sqrt=true", "-shared", "-Xcompiler", "-fPIC", "-I",
                    os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "ultraballpit_b200", "csrc"), "-o",
                    str(out), os.path.join(ROOT, "tests", "cuda", "arith_check.cu")], check=True)
    lib = ctypes.CDLL(str(out))
    lib.arith_check.argtypes = [ctypes.c_float, ctypes.c_float, ctypes.POINTER(ctypes.c_float), ctypes.c_int,
                                ctypes.c_float, ctypes.POINTER(ctypes.c_ulonglong)]
    lib.arith_check.restype = ctypes.c_int
    return lib


@pytest.mark.parametrize("scale", [2.0 ** -100, 2.0 ** -40, 1.0, 2.0 ** 20])
def test_fast_operations_equal_ieee(arith, scale):
    f32 = np.float32
    rng = np.random.default_rng(int(abs(np.log2(scale))) + 1)
    # divisors of every kind of mantissa (all ones, powers of two, their neighbours, random), over the binades of
    # d2 + eta^2 and of density sums
    m = np.concatenate([[1.0, 1.0 + 2.0 ** -23, 2.0 - 2.0 ** -23, 2.0 - 2.0 ** -22], rng.uniform(1.0, 2.0, 28)])
    b = np.concatenate([m * 2.0 ** e for e in (-26, -13, -1, 0, 10, 20)]).astype(f32)
    bad = (ctypes.c_ulonglong * 3)()
    assert arith.arith_check(f32(2.0 ** -100), f32(2.0 ** 60), b.ctypes.data_as(ctypes.POINTER(ctypes.c_float)),
                             len(b), scale, bad) == 0
    assert list(bad) == [0, 0, 0]


def plain(sc, rng):
    pass


def coincident(sc, rng):
    p = sc.particles
    p.x[1], p.y[1], p.z[1] = p.x[0], p.y[0], p.z[0]
    p.x[11], p.y[11], p.z[11] = p.x[10] + np.float32(2e-9), p.y[10], p.z[10]


def close_to_origin(sc, rng):  # neighbours 1e-13 apart, representable near 0
    p = sc.particles
    p.x[0], p.y[0], p.z[0] = 0.0, 0.0, 0.0
    p.x[1], p.y[1], p.z[1] = 1e-13, 0.0, 0.0
    p.x[2], p.y[2], p.z[2] = 0.0, 3e-12, 0.0


def tiny_velocities(sc, rng):
    p = sc.particles
    for a in (p.vx, p.vy, p.vz):
        a[:] = (rng.uniform(-1, 1, len(p)) * 10.0 ** rng.uniform(-42, -8, len(p))).astype(np.float32)


def fast_particles(sc, rng):
    sc.particles.vx[5], sc.particles.vy[6] = 1e6, -3e4


def odd_densities(sc, rng):  # above what the quotients by density sums allow
    sc.particles.density[4] = 2e9


def odd_masses(sc, rng):  # below what they allow, one alone: its density is tiny
    p = sc.particles
    p.mass[3], p.mass[41] = 1e-20, 1e-25
    p.x[41], p.z[41] = 0.07, 0.035


def dense_at_wall(sc, rng):  # more than 128 neighbours, and lists that the walls overflow
    p = sc.particles
    n = len(p) // 2
    for a, lo, hi in ((p.x, 0.001, 0.02), (p.y, 0.001, 0.035), (p.z, 0.001, 0.02)):
        a[:n] = rng.uniform(lo, hi, n).astype(np.float32)


@pytest.mark.parametrize("order", [CELL_ORDER_ROWS, CELL_ORDER_MORTON])
@pytest.mark.parametrize("coef", [(0.02, 2.0), (0.0, 2.0), (1.0, 0.0), (0.0, 0.0), (-0.5, 2.0)])
@pytest.mark.parametrize("change", [plain, coincident, close_to_origin, tiny_velocities, fast_particles, odd_densities,
                                    odd_masses, dense_at_wall])
def test_operands_outside_the_fast_range(change, coef, order):
    if change not in (plain, tiny_velocities) and (coef != (0.02, 2.0) or order != CELL_ORDER_ROWS):
        pytest.skip("one set of coefficients and one order for the states that do not depend on them")
    sc = small_dam_break()
    change(sc, np.random.default_rng(8))
    sc.alpha, sc.beta = coef
    gpu = CudaKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta, cell_order=order)
    cpu = orc.OracleKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta, tier=1, threads=8, pow_mode=1)
    for _ in range(3):
        gpu.step(2e-5)
        cpu.step(2e-5)
        assert_same(gpu.particles(), cpu.particles())
    gpu.close()


@pytest.mark.parametrize("scale", [0.5, 500.0])
def test_large_smoothing_length(scale):
    sc = domain.dam_break(scale, seed=2, block=(8 * scale, 6 * scale, 6 * scale),
                          domain_max=(12 * scale, 6 * scale, 6 * scale), with_sdf=False)
    gpu = CudaKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta)
    cpu = orc.OracleKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta, tier=1, threads=8, pow_mode=1)
    for _ in range(3):
        dt = cpu.compute_timestep(sc.cfl_number)
        gpu.step(dt)
        cpu.step(dt)
        assert_same(gpu.particles(), cpu.particles())
    gpu.close()
