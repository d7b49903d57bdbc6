"""The kernels of a step as programmatic dependents (the handle's own stream) against the plain order (the legacy default
stream): the same state, sums and wall force bit for bit, after steps that follow one another without a pause."""
import ctypes

import numpy as np
import pytest

from lbm_b200 import warmstart as ws
from lbm_b200.kernel import B200Kernel

pytestmark = pytest.mark.gpu
LEGACY_STREAM = 1


def run(shape, precision, solids, open_faces, stream):
    nx, ny, nz = shape
    lattice = ws.channel_lattice(shape)
    if not open_faces:
        lattice.face_boundary = (ctypes.c_int*6)()
        lattice.body_acceleration[0] = 1e-4
    y, z = np.meshgrid(np.arange(ny), np.arange(nz), indexing='xy')
    wall = np.repeat(((y == 0) | (y == ny - 1) | (z == 0) | (z == nz - 1)).ravel(), nx)
    kernel = B200Kernel(lattice, [], np.nonzero(wall)[0] if solids else [], precision, stream=stream)
    for step in range(60):
        kernel.begin_step(step)
        kernel.execute(step)
    return [np.array(kernel.get_fluid_state()), kernel.get_fluid_mach_number()] + [np.array(f) for f in kernel.get_fluid_fields()]


@pytest.mark.parametrize('shape', [(16, 8, 8), (38, 17, 11), (31, 9, 10)])
@pytest.mark.parametrize('precision', ['single', 'half', 'double'])
@pytest.mark.parametrize('solids,open_faces', [(False, False), (True, False), (True, True)])
def test_step_order(shape, precision, solids, open_faces):
    here = run(shape, precision, solids, open_faces, None)
    plain = run(shape, precision, solids, open_faces, LEGACY_STREAM)
    assert all(np.isfinite(a).all() for a in here)
    for a, b in zip(here, plain):
        assert np.array_equal(a, b)
