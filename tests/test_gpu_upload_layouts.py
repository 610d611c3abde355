"""Host samples of every layout reach the device element by element, each from data of its own."""

import pytest
import torch

pytestmark = pytest.mark.gpu

SLOT = 4 << 20


@pytest.mark.parametrize('layout', ['rows', 'transposed', 'every second row', 'offset', 'pinned', 'transposed pinned'])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('nbytes', [64, 2 * SLOT, 5 * SLOT + 4096])
def test_upload_layouts(nbytes, dtype, layout):
    """No tolerance: a copy.  The host memory is overwritten as soon as the call returns where it is pageable."""
    from acoular_b200 import device as D
    n = nbytes // dtype.itemsize // 4
    if layout == 'rows':
        x = torch.randn(n, 4, dtype=dtype)
    elif layout == 'transposed':
        x = torch.randn(4, n, dtype=dtype).t()
    elif layout == 'every second row':
        x = torch.randn(2 * n, 4, dtype=dtype)[::2]
    elif layout == 'offset':
        x = torch.randn(n + 1, 4, dtype=dtype)[1:]
    elif layout == 'pinned':
        x = torch.randn(n, 4, dtype=dtype).pin_memory()
    else:
        x = torch.randn(4, n, dtype=dtype).pin_memory().t()
    kept = x.clone()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        d = D.upload_samples(x, 'cuda')
    if layout.endswith('pinned'):
        side.synchronize()
    x.fill_(7.0)
    torch.cuda.current_stream().wait_stream(side)
    assert d.device.type == 'cuda' and d.dtype == dtype and d.shape == kept.shape
    assert torch.equal(d.cpu(), kept)
