"""The bounded waits of the tensor-core Gram: what a wait that runs out leaves behind is marked, never stale.

The limit is set to 100 ns, far shorter than the bulk copies and MMAs that the waits cover, so waits run out on a normal
input (no fault, no trap, nothing that never finishes).
"""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['tc_tf32', 'tc_bf16x3'])
@pytest.mark.parametrize('M', [33, 150])
def test_abandoned_tiles_are_nan(M, precision):
    """Every entry of the finished and of the accumulated matrix is the full run's, bit for bit, or NaN."""
    from acoular_b200 import _native as N
    from acoular_b200 import device as D
    L = N.lib()
    x = torch.randn(40000, M, device='cuda')
    args = (x, 256, 'Hanning', '50%', precision)
    full = D.csm_finished(*args, 1.0)
    upper, _ = D.csm_upper_accumulate(*args)
    marked = 0
    for _ in range(3):
        out, acc = torch.full_like(full, 7.0), torch.zeros_like(upper)
        prev = L.acb_tc_set_wait_limit_ns(100)
        try:
            D.csm_finished(*args, 1.0, out=out)
            D.csm_upper_accumulate(*args, csm_upper=acc)
        finally:
            L.acb_tc_set_wait_limit_ns(prev)
        for got, want in ((out, full), (acc, upper)):
            bad = torch.isnan(got)
            assert torch.equal(got[~bad], want[~bad])
            marked += int(bad.sum())
    assert marked > 0                                       # the short waits ran out
    assert torch.equal(D.csm_finished(*args, 1.0), full)    # and the device is as before
