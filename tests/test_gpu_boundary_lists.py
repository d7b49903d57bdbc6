"""The pass over regularized walls and open faces on lists that end inside and at the edge of its blocks of 64 nodes,
with odd lattice sizes and every face kind, against the oracle (FP64 1e-12, FP32 1e-5, as the parity tests)."""
import numpy as np
import pytest

import lbm_b200
from lbm_b200 import LBMForce
from oracle import OracleKernel

pytestmark = pytest.mark.gpu


def run(shape, fluctuations, kernel_factory, properties):
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
    force.setFluidFluctuations(fluctuations)
    force.setRandomNumberSeed(7)
    force.setSolidNodes([i + nx*(j + ny*k) for k in range(nz) for j in (0, ny - 1) for i in range(nx)])
    force.setWallScheme(LBMForce.Regularized)
    force.setFaceBoundary(LBMForce.XMin, LBMForce.DensityVelocity if fluctuations else LBMForce.Velocity)
    force.setFaceVelocity(LBMForce.XMin, (0.5, 0.1, 0.0))
    force.setFaceBoundary(LBMForce.XMax, LBMForce.Velocity if fluctuations else LBMForce.Density)
    force.setFaceVelocity(LBMForce.XMax, (0.4, 0.0, 0.1))
    system.addForce(force)
    context = lbm_b200.Context(system, lbm_b200.VerletIntegrator(0.01), kernel_factory, properties)
    context.setPositions([(0.1, 0.7, 0.3)])
    context.integrator.step(12)
    out = force.getFluidState(context), np.array(force.getWallForce(context))
    context.close()
    return out


@pytest.mark.parametrize('precision,fluctuations', [('double', False), ('double', True), ('single', False)])
@pytest.mark.parametrize('shape', [(4, 3, 3), (7, 10, 4), (16, 6, 4), (33, 5, 3)])
def test_boundary_pass_agrees_with_oracle(shape, precision, fluctuations):
    state, wall = run(shape, fluctuations, OracleKernel, None)
    got, got_wall = run(shape, fluctuations, None, {'Precision': precision})
    tolerance = 1e-12 if precision == 'double' else 1e-5
    assert abs(got - state).max() <= tolerance*abs(state).max()
    assert abs(got_wall - wall).max() <= (5 if precision == 'single' else 1)*tolerance*max(1.0, abs(wall).max())
