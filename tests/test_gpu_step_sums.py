"""The sums that one step leaves to the next: with the momentum removed in every step, a dense kernel that starts while the
kernel before it still ends reads the velocity which that one writes.  Steps in programmatic order (the handle's own stream)
against the plain order (the legacy default stream): state, fields, Mach number and wall force bit for bit, on lattices whose
sums the dense kernel's last block forms and on those where a launch of their own does (solid nodes, open faces)."""
import ctypes

import numpy as np
import pytest

from lbm_b200 import warmstart as ws
from lbm_b200.kernel import B200Kernel

pytestmark = pytest.mark.gpu
LEGACY_STREAM = 1


def run(shape, precision, geometry, stream):
    nx, ny, nz = shape
    lattice = ws.channel_lattice(shape)
    if geometry != 'faces':
        lattice.face_boundary = (ctypes.c_int*6)()
        lattice.momentum_removal_frequency = 1
        lattice.body_acceleration[:] = [1e-4, -3e-5, 2e-5]
        lattice.initial_velocity[:] = [0.03, 0.01, -0.02]
    y, z = np.meshgrid(np.arange(ny), np.arange(nz), indexing='xy')
    wall = np.repeat(((y == 0) | (y == ny - 1) | (z == 0) | (z == nz - 1)).ravel(), nx)
    kernel = B200Kernel(lattice, [], [] if geometry == 'periodic' else np.nonzero(wall)[0], precision, stream=stream)
    n = nx*ny*nz
    # A disturbance with no symmetry, so that the removed velocity changes from step to step.
    kernel.set_fluid_state(np.array(kernel.get_fluid_state()) + 1e-3*np.sin(0.7*np.arange(19*n)))
    for step in range(60):
        kernel.begin_step(step)
        kernel.execute(step)
    out = [np.array(kernel.get_wall_force()), np.array(kernel.get_fluid_state()), np.array(kernel.get_fluid_mach_number())]
    out += [np.array(f) for f in kernel.get_fluid_fields()]
    kernel.close()
    return out


@pytest.mark.parametrize('shape', [(16, 8, 8), (38, 17, 11), (31, 9, 10)])
@pytest.mark.parametrize('precision', ['single', 'half', 'double'])
@pytest.mark.parametrize('geometry', ['periodic', 'walls', 'faces'])
def test_sums_of_the_step_before(shape, precision, geometry):
    here = run(shape, precision, geometry, None)
    plain = run(shape, precision, geometry, LEGACY_STREAM)
    assert geometry == 'periodic' or abs(here[0]).max() > 0
    for a, b in zip(here, plain):
        assert np.isfinite(a).all() and np.array_equal(a, b)
