"""The bias's gradient: whole numbers, whose sums are exact in any order, to the last voxel; the same bits at every call;
and, for other values, within the rounding of its order of sums: a thread adds ceil(voxels/(592 lanes)) values one after
another (two at least), a block 8 levels, the sum over the blocks 592/128 in a chain and 2 + 5 levels, so that no value
passes more than 20 additions besides its thread's, each off by 2^-24 of a sum of magnitudes at most.  Volumes of less than
a block, of a few blocks and of all, and channels that do not divide a block's threads."""
import ctypes

import pytest
import torch

from lbm_b200 import warmstart as ws

pytestmark = pytest.mark.gpu

SHAPES = [(1, 8, 1, 1, 1), (1, 16, 3, 5, 7), (2, 24, 9, 31, 33), (1, 160, 8, 8, 16), (1, 256, 20, 17, 19), (1, 512, 4, 6, 5),
          (2, 16, 40, 64, 65)]


def volume(shape, seed, whole):
    g = torch.Generator(device='cuda')
    g.manual_seed(seed)
    t = torch.randint(-3, 4, shape, device='cuda', generator=g) if whole else torch.randn(shape, device='cuda', generator=g)
    return ws._volume(t.to(torch.bfloat16))


@pytest.mark.parametrize('shape', SHAPES)
@pytest.mark.parametrize('relu', [False, True])
def test_bias_sums(shape, relu):
    y = volume(shape, 1, False) if relu else None
    voxels, lanes = shape[0]*shape[2]*shape[3]*shape[4], 256//(shape[1]//8)
    for whole in (True, False):
        dy = volume(shape, 2, whole)
        out, db = ws.relu_bias_grad(dy, y)
        ref = out.double().sum(dim=(0, 2, 3, 4))
        if whole:
            assert torch.equal(db.double(), ref)
        else:
            steps = max(2, -(-voxels//(592*lanes))) + 20
            assert ((db.double() - ref).abs() <= steps*2.0**-24*out.double().abs().sum(dim=(0, 2, 3, 4))).all()
        for _ in range(5):
            assert torch.equal(ws.relu_bias_grad(dy, y)[1], db)


def test_the_form_without_scratch_adds_the_same():
    dy = volume(SHAPES[2], 3, False)
    _, expected = ws.relu_bias_grad(dy)
    db = torch.zeros(24, device='cuda')
    lib = ws._lib()
    voxels = dy.numel()//24
    for times in (1, 2):
        assert lib.lbm_net_relu_bias_grad(dy.data_ptr(), None, None, db.data_ptr(), voxels, 24, ws._stream()) == 0
        assert torch.equal(db, times*expected)
    assert lib.lbm_net_relu_bias_grad(dy.data_ptr(), None, None, db.data_ptr(), voxels, 20, ws._stream()) != 0
    assert lib.lbm_net_relu_bias_scratch(ctypes.c_longlong(voxels), 20) == 0
