"""The dense kernels that take pairs and quads of nodes in the order of the nodes, on lattices whose rows end inside a warp,
whose last block is full, partly filled or holds a single row: FP32 against the oracle (1e-5, as the parity tests), 16-bit
storage against FP32 within the rounding of its stores (a step rounds a population by 2^-10 of the largest at most, and
the linear collision passes less than three times that on)."""
import numpy as np
import pytest

import lbm_b200
from lbm_b200 import LBMForce
from oracle import OracleKernel

pytestmark = pytest.mark.gpu
STEPS = 12


def run(shape, walls, kernel_factory, properties):
    nx, ny, nz = shape
    system = lbm_b200.System()
    system.setDefaultPeriodicBoxVectors((nx*0.5, 0, 0), (0, ny*0.5, 0), (0, 0, nz*0.5))
    system.addParticle(1.0)
    force = LBMForce()
    force.setGridSize(nx, ny, nz)
    force.setKinematicViscosity((0.8 - 0.5)/3*0.25/0.01)
    force.setBodyAcceleration((0.5, -0.2, 0.1))
    force.setInitialFluidVelocity((0.5, 0.2, -0.3))
    force.setFluidMomentumRemovalFrequency(0)
    if walls:
        force.setSolidNodes([i + nx*(j + ny*k) for k in range(nz) for j in (0, ny - 1) for i in range(nx)])
    system.addForce(force)
    context = lbm_b200.Context(system, lbm_b200.VerletIntegrator(0.01), kernel_factory, properties)
    context.setPositions([(0.1, 0.7, 0.3)])
    state = force.getFluidState(context)
    state = np.array(state).reshape(19, nz, ny, nx)
    # A disturbance with no symmetry, so that every node differs.
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing='ij')
    state *= 1 + 0.9*np.sin(1.3*x + 2.1*y + 0.7*z + np.arange(19)[:, None, None, None])
    force.setFluidState(context, state.ravel())
    context.integrator.step(STEPS)
    out = np.array(force.getFluidState(context)).reshape(19, nz, ny, nx)
    context.close()
    return out


@pytest.mark.parametrize('shape', [(8, 4, 3), (16, 8, 4), (34, 5, 3), (36, 7, 9), (62, 9, 5), (132, 6, 3)])
@pytest.mark.parametrize('walls', [False, True])
def test_node_order(shape, walls):
    def here(precision):
        return run(shape, walls, None, {'Precision': precision})

    ref = run(shape, walls, OracleKernel, None)
    single = here('single')
    scale = np.abs(ref).max()
    assert np.abs(single - ref).max() <= 1e-5*scale
    for precision in ('half', 'bfloat16'):
        bound = STEPS*3*(2.0**-10 if precision == 'half' else 2.0**-7)
        assert np.abs(here(precision) - single).max() <= bound*scale
