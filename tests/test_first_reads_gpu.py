"""Reads of the particle state before and after the page-locked staging is made
(once 40 MiB have been read without it), for sizes on both sides of what is
read in pageable pieces (2 MiB, 42,799 particles of 49 bytes) and of a piece."""
import time

import numpy as np
import pytest

from test_readback_gpu import check, kernel, state

pytestmark = pytest.mark.gpu


@pytest.fixture
def staged():
    """A handle that has been read often enough for the staging to be there, as long as it lives."""
    p = state(300001)
    k = kernel(p)
    for _ in range(5):
        k._cache = None
        check(k.particles(), p)
    yield k
    k.close()


SIZES = [1, 5, 5349, 5350, 5351, 21399, 21400, 42799, 42800, 171196, 171200, 300001]


@pytest.mark.parametrize("n", SIZES)
def test_first_read(n):
    p = state(n)
    k = kernel(p)
    check(k.particles(), p)
    k.close()


@pytest.mark.parametrize("n", SIZES)
def test_read_through_the_staging(staged, n):
    p = state(n, 2)
    k = kernel(p)
    for _ in range(2):
        k._cache = None
        check(k.particles(), p)
    k.close()


def test_staging_grows_with_the_reads():
    small, large = state(30000), state(200000)
    a, b = kernel(small), kernel(large)
    for k, p, reads in ((a, small, 40), (b, large, 8), (a, small, 2)):
        for _ in range(reads):
            k._cache = None
            check(k.particles(), p)
    a.close()
    b.close()


def test_a_single_read_does_not_pay_for_the_staging():
    """A simulation created, read once and destroyed: making and giving back the staging took 1.5 ms or more of it."""
    p = state(2000)
    kernel(p).particles()  # the process's first
    took = []
    for _ in range(10):
        k = kernel(p)
        k.compute_timestep()
        t0 = time.perf_counter()
        k.particles()
        took.append(time.perf_counter() - t0)
        k.close()
    assert np.min(took) < 0.75e-3
