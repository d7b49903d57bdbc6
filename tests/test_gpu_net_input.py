"""The network's input for every kind of inlet and mask that torch takes: the forms that the kernel does not serve give what
torch's assignments give, the others the same as those."""
import numpy as np
import pytest
import torch

from lbm_b200 import warmstart as ws

pytestmark = pytest.mark.gpu


def by_torch(masks, inlet):
    """The input as a float volume, rounded once."""
    nz, ny, nx = masks[0].shape
    x = torch.zeros((len(masks), ws.IN_CHANNELS, nz, ny, nx), device='cuda')
    for i, m in enumerate(masks):
        x[i, 0], x[i, 1] = m.float(), inlet/ws.INLET_SCALE
        x[i, 2] = torch.linspace(0, 1, nx, device='cuda').view(1, 1, nx)
        x[i, 3] = torch.linspace(0, 1, ny, device='cuda').view(1, ny, 1)
        x[i, 4] = torch.linspace(0, 1, nz, device='cuda').view(nz, 1, 1)
    return x.to(torch.bfloat16)


@pytest.mark.parametrize('inlet', [0.013, 1, np.float64(0.017), torch.tensor(0.013),
                                   'device', 'profile'])
def test_inlets(inlet):
    nz, ny, nx = 5, 6, 7
    if isinstance(inlet, str):
        inlet = torch.tensor(0.021, device='cuda') if inlet == 'device' else torch.linspace(0, 0.02, ny, device='cuda').view(ny, 1)
    g = torch.Generator(device='cuda')
    g.manual_seed(1)
    masks = [torch.rand((nz, ny, nx), device='cuda', generator=g) < 0.4 for _ in range(2)]
    got = ws.network_input(masks, inlet)
    assert torch.equal(got, by_torch(masks, inlet)) and got.is_contiguous(memory_format=torch.channels_last_3d)


def test_empty_masks():
    mask = torch.zeros((0, 4, 3), device='cuda', dtype=torch.bool)
    assert tuple(ws.network_input([mask]).shape) == (1, ws.IN_CHANNELS, 0, 4, 3)
