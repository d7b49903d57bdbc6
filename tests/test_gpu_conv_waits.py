"""Waits for the tensor cores that run out, in every form of the convolutions (weights held, one channel group, streamed,
gathered; weight gradients of all dz at once and one by one): with a limit of 0 every role of a block gives up at its first
wait and the timeout is reported; with limits that some waits outlast and others do not, roles give up one after another,
and the call ends either way.  Afterwards the same call gives its result again.  Volumes that end inside a tile, so that
some lanes of the reading warps have nothing to store; small whole numbers, whose sums are exact in any order."""
import pytest
import torch

from lbm_b200 import warmstart as ws
from lbm_b200.abi import LBM_ERR_DEVICE_TIMEOUT, LbmError

pytestmark = pytest.mark.gpu


def integers(shape, seed):
    g = torch.Generator(device='cuda')
    g.manual_seed(seed)
    return torch.randint(-2, 3, shape, device='cuda', generator=g).to(torch.bfloat16)


def forward(cin, cout, shape):
    x, w = ws._volume(integers((2, cin) + shape, 1)), integers((cout, 27, cin), 2)
    return lambda: ws.conv3d_forward(x, w, None, False)


def gradient(cin, cout, shape):
    x, dy = ws._volume(integers((2, cin) + shape, 3)), ws._volume(integers((2, cout) + shape, 4))
    return lambda: ws.conv3d_weight_grad(x, dy)


@pytest.mark.parametrize('call,cin,cout', [(forward, 8, 16), (forward, 16, 32), (forward, 160, 160), (forward, 24, 16),
                                           (gradient, 16, 16), (gradient, 48, 64)])
def test_waits_that_run_out(call, cin, cout):
    lib = ws._lib()
    run = call(cin, cout, (9, 21, 13))
    expected = run()
    ws.conv_status()
    try:
        for limit in (0, 1, 4, 16, 64, 256):
            assert lib.lbm_conv3d_set_wait_limit(limit) == 0
            run()
            try:
                ws.conv_status()
                assert limit > 0
            except LbmError as failure:
                assert failure.status == LBM_ERR_DEVICE_TIMEOUT
    finally:
        assert lib.lbm_conv3d_set_wait_limit(-1) == 0
    again = run()
    ws.conv_status()
    assert torch.equal(again, expected)
