"""Fields handed to the kernel while torch is still computing them on its own stream."""
import numpy as np
import pytest
import torch

import lbm_b200
from lbm_b200 import LBMForce

pytestmark = pytest.mark.gpu


def test_equilibrium_waits_for_the_stream_of_its_fields():
    n = 16
    force = LBMForce()
    force.setGridSize(n, n, n)
    force.setFluidDensity(1.0)
    force.setKinematicViscosity(0.1)
    kernel = lbm_b200.B200Kernel(force.latticeParameters(np.array([n, n, n], dtype=float), 1.0, np.ones(1)), [], [], 'double')
    density = torch.full((n**3,), 7.0, device='cuda', dtype=torch.float64)
    velocity = torch.full((n**3, 3), 7.0, device='cuda', dtype=torch.float64)
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)      # some 50 ms of the stream's time before the fields get their values
    density.fill_(1.01)
    velocity.fill_(0.02)
    kernel.set_fluid_equilibrium(density, velocity, strain=False)
    rho, u = kernel.get_fluid_fields()
    assert abs(rho - 1.01).max() <= 1e-12 and abs(u - 0.02).max() <= 1e-12
    kernel.close()
