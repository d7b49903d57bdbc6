"""Volumes and weights that are views into a larger buffer at an address that is no multiple of 16 bytes: every entry of the
warm start's network gives what it gives for a copy of them."""
import pytest
import torch

from lbm_b200 import warmstart as ws

pytestmark = pytest.mark.gpu


def pair(shape, seed, channels_last=True):
    """A tensor, and one of the same values that starts 2 bytes into its buffer."""
    g = torch.Generator(device='cuda')
    g.manual_seed(seed)
    order = shape[:1] + shape[2:] + shape[1:2] if channels_last else shape
    flat = torch.randn(order, device='cuda', generator=g).to(torch.bfloat16).flatten()
    buffer = torch.empty(flat.numel() + 1, device='cuda', dtype=torch.bfloat16)
    buffer[1:] = flat

    def as_volume(t):
        t = t.view(order)
        return t.permute(0, 4, 1, 2, 3) if channels_last else t
    a, b = as_volume(flat), as_volume(buffer[1:])
    assert a.data_ptr() % 16 == 0 and b.data_ptr() % 16 == 2
    return a, b


def test_unaligned_views():
    x, xu = pair((1, 16, 4, 6, 10), 1)
    dy, dyu = pair((1, 32, 4, 6, 10), 2)
    skip, skipu = pair((1, 8, 8, 12, 20), 3)
    w, wu = pair((32, 27, 16), 4, channels_last=False)
    assert torch.equal(ws.conv3d_forward(xu, wu), ws.conv3d_forward(x, w))
    assert torch.equal(ws.conv3d_input_grad(dyu, wu), ws.conv3d_input_grad(dy, w))
    assert torch.allclose(ws.conv3d_weight_grad(xu, dyu), ws.conv3d_weight_grad(x, dy), rtol=0, atol=1e-3)
    assert torch.equal(ws.Pool2.apply(xu), ws.Pool2.apply(x))
    assert torch.equal(ws.UpsampleConcat.apply(xu, skipu), ws.UpsampleConcat.apply(x, skip))
    for y, yu in ((None, None), pair((1, 32, 4, 6, 10), 5)):
        for a, b in zip(ws.relu_bias_grad(dyu, yu), ws.relu_bias_grad(dy, y)):
            assert torch.equal(a, b)


@pytest.mark.parametrize('relu', [False, True])
def test_unaligned_output_gradient(relu):
    x, _ = pair((1, 16, 4, 6, 10), 6)
    dy, dyu = pair((1, 32, 4, 6, 10), 7)
    grads = []
    for g in (dy, dyu):
        leaves = [x.detach().clone().requires_grad_(True),
                  torch.linspace(-1, 1, 32*27*16, device='cuda').view(32, 27, 16).requires_grad_(True),
                  torch.zeros(32, device='cuda', requires_grad=True)]
        ws.Conv3dFunction.apply(*leaves, relu).backward(g)
        grads.append([t.grad for t in leaves])
    for a, b in zip(*grads):
        # The weight's gradient is added up by atomics, whose order is not fixed.
        assert torch.allclose(a, b, rtol=0, atol=1e-5*float(a.abs().max()))
