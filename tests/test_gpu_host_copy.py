"""Fields and state read back by one thread and by several (lattices around the size at which they share the copy, and with
a last chunk that is not full): the fields are those of the state, and a state that is read, set and read again is the
same bit for bit."""
import numpy as np
import pytest

import lbm_b200
from lbm_b200 import LBMForce

pytestmark = pytest.mark.gpu

WEIGHTS = np.array([1/3] + [1/18]*6 + [1/36]*12)
VELOCITIES = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
                       (1, -1, 0), (-1, 1, 0), (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1), (1, 0, 1), (-1, 0, -1),
                       (-1, 0, 1), (1, 0, -1)])


@pytest.mark.parametrize('shape', [(5, 3, 4), (64, 64, 63), (64, 64, 65), (101, 67, 59)])
def test_fields_are_those_of_the_state(shape):
    nx, ny, nz = shape
    n = nx*ny*nz
    force = LBMForce()
    force.setGridSize(nx, ny, nz)
    force.setFluidDensity(1.0)
    force.setKinematicViscosity(0.1)
    kernel = lbm_b200.B200Kernel(force.latticeParameters(np.array(shape, dtype=float), 1.0, np.ones(1)), [], [], 'double')
    rng = np.random.default_rng(nx)
    state = (1e-3*WEIGHTS[:, None]*rng.standard_normal((19, n))).ravel()
    kernel.set_fluid_state(state)
    assert np.array_equal(kernel.get_fluid_state(), state)
    density, velocity = kernel.get_fluid_fields()
    f = state.reshape(19, n)
    rho = 1.0 + f.sum(axis=0)
    u = (VELOCITIES.T @ f).T/rho[:, None]
    assert abs(density - rho).max() <= 1e-13
    assert abs(velocity - u).max() <= 1e-13
    kernel.close()
