"""The length of the weight gradient's sums on the tensor core, which truncates them.

The output gradient is 1 in a few blocks of voxels and 0 elsewhere; in every run of 16 x-neighbours the input is `big` at 15
voxels and 1 at one, so an MMA (16 voxels) adds c = 15 big + 1, an odd number (14 big + 1 at the volume's edges).  A sum of
`most` MMAs stays below 2^24 and is exact; one of more is truncated, and an entry comes out too small.  What the atomics add
up is exact in any order: the finished sums are even multiples of c or below 2^24, and their totals below 2^25.  So with
sums of at most `most` MMAs, as the division of the work (planGradient) states, every entry is exact.

The blocks of the larger volume are those of two items that one block of threads takes in turn on 148 SMs: 6 rows of 8 and 4
planes, 24 MMAs, then 32."""
import numpy as np
import pytest
import torch

from lbm_b200 import warmstart as ws
import conv_oracle

pytestmark = pytest.mark.gpu


def volume(a):
    return ws._volume(torch.as_tensor(a, dtype=torch.float32).to(torch.bfloat16).permute(0, 4, 1, 2, 3).cuda())


@pytest.mark.parametrize('shape,blocks,big', [
    ((2, 8, 16), [(slice(0, 2), slice(0, 8), slice(0, 16))], 2.0**17),
    ((64, 62, 64), [(slice(4, 8), slice(56, 62), slice(0, 16)), (slice(24, 28), slice(32, 40), slice(0, 16))], 2.0**15)])
def test_sums_are_no_longer_than_stated(shape, blocks, big):
    x = np.full((1,) + shape + (16,), big)
    x[:, :, :, 5::16] = 1.0
    dy = np.zeros((1,) + shape + (16,))
    for block in blocks:
        dy[(0,) + block] = 1.0
    got = ws.conv3d_weight_grad(volume(x), volume(dy))
    ws.conv_status()
    assert np.array_equal(got.cpu().numpy(), conv_oracle.conv3d_weight_grad(x, dy))
