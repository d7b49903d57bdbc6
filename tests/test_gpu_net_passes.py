"""The network's passes between the convolutions against the same passes of torch (float32 on the same BF16 values,
rounded once): bit for bit, at odd sizes, single planes and channel counts that do not divide a block; the bias's gradient
(an FP32 sum in another order) within the sum of magnitudes times voxels 2^-24."""
import numpy as np
import pytest
import torch

from lbm_b200 import warmstart as ws

pytestmark = pytest.mark.gpu

SHAPES = [(1, 16, 2, 2, 2), (2, 16, 6, 4, 10), (1, 160, 4, 2, 6), (1, 8, 16, 8, 130), (1, 24, 5, 7, 9)]


def volume(shape, seed):
    g = torch.Generator(device='cuda')
    g.manual_seed(seed)
    return ws._volume(torch.randn(shape, device='cuda', generator=g).to(torch.bfloat16))


@pytest.mark.parametrize('shape', SHAPES)
def test_pool_and_its_gradient(shape):
    x = volume(shape, 1).requires_grad_(True)
    y = ws.Pool2.apply(x)
    ref_x = x.detach().float().requires_grad_(True)
    ref = torch.nn.functional.avg_pool3d(ref_x, 2)
    assert torch.equal(y, ref.to(torch.bfloat16))
    dy = volume(tuple(y.shape), 2)
    y.backward(dy)
    ref.backward(dy.float())
    assert torch.equal(x.grad, ref_x.grad.to(torch.bfloat16))


@pytest.mark.parametrize('shape,skip', [(SHAPES[0], 16), (SHAPES[1], 32), (SHAPES[2], 64), (SHAPES[4], 8)])
def test_upsampling_with_the_skip_and_its_gradients(shape, skip):
    n, c, d, h, w = shape
    x, s = volume(shape, 3).requires_grad_(True), volume((n, skip, 2*d, 2*h, 2*w), 4).requires_grad_(True)
    y = ws.UpsampleConcat.apply(x, s)
    ref_x, ref_s = x.detach().float().requires_grad_(True), s.detach().float().requires_grad_(True)
    ref = torch.cat([torch.nn.functional.interpolate(ref_x, scale_factor=2, mode='nearest'), ref_s], dim=1)
    assert torch.equal(y, ref.to(torch.bfloat16))
    dy = volume(tuple(y.shape), 5)
    y.backward(dy)
    ref.backward(dy.float())
    assert torch.equal(s.grad, ref_s.grad.to(torch.bfloat16))
    # A sum of 8 in FP32, rounded once; torch may add in another order.
    assert (x.grad.float() - ref_x.grad).abs().max() <= 2.0**-8*ref_x.grad.abs().max()
    with pytest.raises(RuntimeError):
        ws.UpsampleConcat.apply(x, s[:, :, :-1])


@pytest.mark.parametrize('shape', SHAPES + [(1, 256, 3, 3, 3)])
@pytest.mark.parametrize('relu', [False, True])
def test_relu_gradient_and_bias_sums(shape, relu):
    dy, y = volume(shape, 6), volume(shape, 7)
    y[:, :, 0, 0, 0] = 0.0
    y[0, 1, 0, 0, 1] = float('nan')
    out, db = ws.relu_bias_grad(dy, y if relu else None)
    ref = dy*(y > 0).to(dy.dtype) if relu else dy
    assert torch.equal(out, ref)
    count = dy.numel()//shape[1]
    bound = dy.float().abs().sum(dim=(0, 2, 3, 4))*count*2.0**-24 + 1e-30
    assert ((db - ref.double().sum(dim=(0, 2, 3, 4))).abs() <= bound).all()


def test_network_input_is_that_of_torch():
    rng = np.random.default_rng(3)
    for shape in ((3, 5, 7), (64, 32, 48)):
        masks = [torch.as_tensor(rng.random(shape) < 0.3, device='cuda') for _ in range(2)]
        got = ws.network_input(masks, 0.013)
        ref = ws.network_input([m.float() for m in masks], 0.013)
        assert torch.equal(got, ref) and got.is_contiguous(memory_format=torch.channels_last_3d)


@pytest.mark.parametrize('sizes', [[(16, 8)], [(48, 40), (16, 16), (160, 224), (20, 3)], [(16, 33)]*33])
def test_packed_weights(sizes):
    g = torch.Generator(device='cuda')
    g.manual_seed(8)
    weights = [torch.randn((cout, 27, cin), device='cuda', generator=g) for cout, cin in sizes]
    transposed = [i % 2 == 0 for i in range(len(sizes))]
    for w, t, (w16, wt) in zip(weights, transposed, ws.pack_weights(weights, transposed)):
        ref = w.to(torch.bfloat16)
        assert torch.equal(w16, ref.flatten())
        assert (wt is not None) == t
        if t:
            assert torch.equal(wt, ref.flip(1).permute(2, 1, 0).flatten())
    assert ws.pack_weights([weights[0].transpose(0, 2)], [False]) is None or sizes[0][0] == sizes[0][1]
    assert ws.pack_weights([weights[0].double()], [False]) is None
