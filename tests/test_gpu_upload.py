"""Host samples staged to the device: the bytes arrive, whatever the size, type, layout, stream and thread."""

import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

SLOT = 4 << 20


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('nbytes', [64, 2 * SLOT - 8, 2 * SLOT, 2 * SLOT + 8, 3 * SLOT, 5 * SLOT + 4096, 7 * SLOT - 16])
def test_upload_is_the_same_bytes(nbytes, dtype):
    """Around the smallest staged size and around whole numbers of slots (no tolerance: a copy)."""
    from acoular_b200 import device as D
    n = nbytes // dtype.itemsize // 4 * 4
    x = torch.randn(n // 4, 4, dtype=dtype)
    for y in (x, x.t(), x[::2]):
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            d = D.upload_samples(y, 'cuda')
        kept, y = y.clone(), y.fill_(7.0)   # the host memory is free again once the call returns
        torch.cuda.current_stream().wait_stream(side)
        assert d.device.type == 'cuda' and d.dtype == dtype
        assert torch.equal(d.cpu(), kept)


def test_upload_from_several_threads():
    from acoular_b200 import device as D
    xs = [torch.full((3 * SLOT // 8 + 5,), float(i), dtype=torch.float64) for i in range(4)]
    out = [None] * len(xs)

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            out[i] = D.upload_samples(xs[i], 'cuda')
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(xs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for x, d in zip(xs, out):
        assert torch.equal(d.cpu(), x)
