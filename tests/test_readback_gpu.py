"""Reads of the particle state through the page-locked staging: sizes around a
piece and around the several-thread path, page-locked destinations (direct
copies), readers in several threads, and handles that come and go."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from ultraballpit_b200.kernel import CudaKernel, SphParticlesMut, load_library
from ultraballpit_b200.particles import PARTICLE_FIELDS, ParticleArrays

pytestmark = pytest.mark.gpu


def state(n, seed=1):
    rng = np.random.default_rng(seed)
    p = ParticleArrays.from_positions(*rng.uniform(0.0, 1.0, (3, n)), 1.0)
    for f in PARTICLE_FIELDS[3:]:
        getattr(p, f)[:] = rng.uniform(0.5, 2.0, n).astype(np.float32)
    p.fluid_type[:] = rng.integers(0, 2, n)
    return p


def kernel(p):
    return CudaKernel(p, None, 0.02, (0.0, 0.0, -9.81), 20.0, 0.25, 0.0, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0))


def check(got, want):
    for f in PARTICLE_FIELDS:
        np.testing.assert_array_equal(getattr(got, f), getattr(want, f))
    np.testing.assert_array_equal(got.fluid_type, want.fluid_type)


# one piece is 1 MiB of 49-byte particles; from 8 MiB on four threads read
@pytest.mark.parametrize("n", [1, 5, 1000, 21399, 21400, 42799, 171196, 171200, 300001])
def test_reads_what_was_written(n):
    p = state(n)
    k = kernel(p)
    check(k.particles(), p)
    k._cache = None
    check(k.particles(), p)
    k.close()


def test_page_locked_destination():
    p = state(50000)
    k = kernel(p)
    bufs = {f: torch.zeros(50000, dtype=torch.float32).pin_memory() for f in PARTICLE_FIELDS}
    ft = torch.zeros(50000, dtype=torch.uint8).pin_memory()
    fp, up = C.POINTER(C.c_float), C.POINTER(C.c_uint8)
    out = SphParticlesMut(50000, *[C.cast(bufs[f].data_ptr(), fp) for f in PARTICLE_FIELDS],
                          C.cast(ft.data_ptr(), up))
    assert load_library().sph_read_particles(k._h, C.byref(out)) == 0
    for f in PARTICLE_FIELDS:
        np.testing.assert_array_equal(bufs[f].numpy(), getattr(p, f))
    np.testing.assert_array_equal(ft.numpy(), p.fluid_type)
    k.close()


def test_readers_in_threads_while_handles_come_and_go():
    errors = []

    def work(seed):
        try:
            for r in range(4):
                p = state((3000, 60000, 200000)[(seed + r) % 3], seed * 10 + r)
                k = kernel(p)
                for _ in range(3):
                    k._cache = None
                    check(k.particles(), p)
                k.close()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(repr(e)[:300])

    ts = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert errors == []
