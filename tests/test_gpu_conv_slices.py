"""The convolutions at the sizes where their division of the work changes, against the float64 oracle: columns of
8 x 16 voxels and one more or fewer, runs of planes with a remainder, one channel group and weights that are held,
streamed or split over blocks of output channels.

Tolerance: the inputs are BF16, the products exact in FP32 and their sum off by less than 27 cin 2^-24 of the sum of
magnitudes, so the BF16 rounding of the output (2^-9 of the element) is what remains: 2^-8 of the largest output."""
import numpy as np
import pytest
import torch

from lbm_b200 import warmstart as ws
import conv_oracle

pytestmark = pytest.mark.gpu


def rounded(a):
    return torch.as_tensor(a, dtype=torch.float32).to(torch.bfloat16).float().numpy().astype(np.float64)


def volume(a):
    return ws._volume(torch.as_tensor(a, dtype=torch.float32).to(torch.bfloat16).permute(0, 4, 1, 2, 3).cuda())


@pytest.mark.parametrize('n,shape,cin,cout', [
    (1, (1, 1, 1), 16, 16), (1, (3, 16, 8), 16, 16), (1, (9, 17, 9), 8, 16), (2, (8, 15, 7), 8, 32),
    (1, (17, 16, 16), 32, 48), (1, (3, 5, 9), 96, 32), (1, (2, 4, 3), 224, 64), (1, (3, 8, 16), 160, 160),
    (1, (2, 9, 5), 240, 16), (1, (2, 3, 4), 24, 16), (1, (4, 4, 4), 64, 256), (3, (5, 33, 20), 16, 16)])
def test_forward_at_the_edges_of_its_tiles(n, shape, cin, cout):
    rng = np.random.default_rng(cin + 3*cout + shape[2])
    x = rounded(rng.standard_normal((n,) + shape + (cin,)))
    w = rounded(rng.standard_normal((cout, 27, cin))*0.1)
    b = rng.standard_normal(cout).astype(np.float32)
    y = ws.conv3d_forward(volume(x), torch.as_tensor(w).to(torch.bfloat16).cuda(), torch.as_tensor(b).cuda(), False)
    ws.conv_status()
    ref = conv_oracle.conv3d_forward(x, w, b, False)
    got = y.float().permute(0, 2, 3, 4, 1).cpu().numpy()
    assert abs(got - ref).max() <= 2.0**-8*abs(ref).max()


@pytest.mark.parametrize('n,shape,cin,cout', [
    (1, (1, 1, 1), 16, 16), (1, (4, 8, 16), 8, 16), (2, (5, 9, 17), 16, 32), (1, (3, 7, 15), 48, 48),
    (1, (9, 17, 33), 40, 16), (1, (3, 9, 18), 88, 64), (1, (2, 5, 20), 224, 160), (1, (4, 3, 5), 24, 112),
    (1, (21, 40, 35), 16, 16)])
def test_weight_gradient_at_the_edges_of_its_tiles(n, shape, cin, cout):
    """FP32 sums of exact products, cut every 48 MMAs of 16 voxels at most: 48 truncations of 2^-24 and the atomics'
    rounding, below 1e-5 of the largest entry."""
    rng = np.random.default_rng(5*cin + cout + shape[2])
    x = rounded(rng.standard_normal((n,) + shape + (cin,)))
    dy = rounded(rng.standard_normal((n,) + shape + (cout,)))
    g = ws.conv3d_weight_grad(volume(x), volume(dy))
    ws.conv_status()
    ref = conv_oracle.conv3d_weight_grad(x, dy)
    assert abs(g.cpu().numpy() - ref).max() <= 1e-5*abs(ref).max()
