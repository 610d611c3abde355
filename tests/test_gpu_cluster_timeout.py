"""The bounded waits between the CTAs of a cluster: where one runs out the result is marked, never a plausible number.

The limit is set to 100 ns, far shorter than the steps that the waits cover, so waits run out on a normal input (no fault,
no trap, nothing that never finishes), and in any CTA of a cluster.
"""

import contextlib

import pytest
import torch

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def short_waits():
    from acoular_b200 import _native as N
    prev = N.lib().acb_tc_set_wait_limit_ns(100)
    try:
        yield
    finally:
        torch.cuda.synchronize()
        N.lib().acb_tc_set_wait_limit_ns(prev)


def test_damas_marks_the_bin():
    """Each bin is the full run's, bit for bit, or NaN throughout.  The grid is large, so that the first CTA waits some
    microseconds for the sums of every step (shorter waits end within the hardware's own suspension)."""
    from acoular_b200 import device as D
    B, G = 2, 10000
    A = torch.rand(B, G, G, dtype=torch.float64, device='cuda').div_(G)
    A.diagonal(dim1=1, dim2=2).fill_(1.0)
    y = torch.rand(B, G, dtype=torch.float64, device='cuda')
    full = D.damas_gauss_seidel(A, y, 2, 1.0, cta_per_bin=4)
    assert torch.isfinite(full).all()
    marked = 0
    for _ in range(3):
        with short_waits():
            got = D.damas_gauss_seidel(A, y, 2, 1.0, cta_per_bin=4)
        for b in range(B):
            bad = torch.isnan(got[b])
            assert bad.all() or torch.equal(got[b], full[b])
            marked += int(bad.all())
    assert marked > 0
    assert torch.equal(D.damas_gauss_seidel(A, y, 2, 1.0, cta_per_bin=4), full)   # and the device is as before
