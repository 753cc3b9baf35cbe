"""Edges of the forms that the neighbour kernels take by size (SPH_GROUP_LANES
sets the lanes per particle): instances without particles, particles in
neighbourhoods past the scan's masks, coefficients and densities outside the
ordinary, and the paths taken only by large grids or without a boundary list."""
import numpy as np
import pytest

from ultraballpit_b200.kernel import CudaBatch

from test_group_forms_gpu import first
from test_parity_gpu import small_dam_break

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
