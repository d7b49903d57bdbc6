"""The dense kernels in row tiles and in the order of the nodes.  A node's step does not depend on the split, so two 16-bit
runs of which one takes row tiles (a momentum removal is set, at a step that is not reached) and the other the nodes' order
(none is set) give the same state and positions bit for bit (not the step's sums, whose order the split sets): quads and
pairs, several tiles along a row and rows that end inside one, solid nodes, walls of both schemes, fluctuations and
particles.  FP32 without solid nodes takes row tiles on lattices above 2^21 nodes: there against the oracle, with the momentum
removed in every step and without (1e-5, as the parity tests)."""
import numpy as np
import pytest

from oracle import OracleKernel
from test_gpu_paired import wide_case

pytestmark = pytest.mark.gpu
FAR = 100000


def run(shape, walls, fluct, particles, precision, removal, steps=30):
    context, force = wide_case(shape, walls, fluct, particles, None, {'Precision': precision}, removal=removal)
    context.step_count = 1      # step 0 would remove the momentum
    context.integrator.step(steps)
    result = np.array(force.getFluidState(context)), context.positions.copy()
    context.close()
    return result


@pytest.mark.parametrize('precision', ['half', 'bfloat16'])
@pytest.mark.parametrize('shape,walls,fluct,particles', [
    ((256, 6, 3), 'periodic', False, 0), ((132, 5, 4), 'periodic', False, 3), ((64, 13, 5), 'walls', False, 3),
    ((128, 9, 4), 'regularized', False, 0), ((130, 9, 4), 'walls', False, 2), ((66, 7, 5), 'periodic', False, 0),
    ((128, 9, 4), 'regularized', True, 2), ((70, 12, 3), 'periodic', True, 0), ((6, 9, 5), 'walls', True, 2)])
def test_row_tiles_are_bitwise_the_node_order(shape, walls, fluct, particles, precision):
    tiles = run(shape, walls, fluct, particles, precision, FAR)
    nodes = run(shape, walls, fluct, particles, precision, 0)
    for a, b in zip(tiles, nodes):
        assert np.isfinite(a).all() and np.array_equal(a, b)


@pytest.mark.parametrize('removal,fluct', [(0, False), (1, False), (1, True)])
def test_fp32_row_tiles_of_a_large_lattice_agree_with_oracle(removal, fluct):
    states = []
    for factory, props in ((OracleKernel, None), (None, {'Precision': 'single'})):
        context, force = wide_case((130, 130, 126), 'periodic', fluct, 0, factory, props, removal=removal)
        context.integrator.step(3)
        states.append(np.array(force.getFluidState(context)))
        context.close()
    ref, got = states
    assert abs(got - ref).max() <= 1e-5*abs(ref).max()
