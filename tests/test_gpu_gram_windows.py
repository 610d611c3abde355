"""Sums over a few windows, around the 16 windows of a stage: all at once, one at a time, added to and finished."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['complex128', 'complex64'])
@pytest.mark.parametrize('K', [1, 2, 3, 4, 5, 13, 15, 16, 17, 20, 21, 33])
@pytest.mark.parametrize('M', [2, 17, 33, 70])
def test_windows_together_and_one_by_one(M, K, precision):
    """An element is one chain of FMAs over the windows, so the bits are the same however they are grouped."""
    from acoular_b200 import device as D
    N = 32
    x = torch.randn((K + 1) * N // 2, M, dtype=torch.float64, device='cuda')
    args = (x, N, 'Hanning', '50%', precision)
    up, n = D.csm_upper_accumulate(*args)
    assert n == K
    one = torch.zeros_like(up)
    for w in range(K):
        D.csm_upper_accumulate(*args, csm_upper=one, first_window=w, windows=1)
    assert torch.equal(up, one)
    assert torch.equal(D.csm_finished(*args, 0.75), D.csm_finalize(up, 0.75))


@pytest.mark.parametrize('precision', ['tc_tf32', 'tc_bf16x3'])
@pytest.mark.parametrize('K', [1, 32, 33, 70])
@pytest.mark.parametrize('M', [1, 15, 64, 65, 130])
def test_tensor_core_sums_added_and_finished(M, K, precision):
    """Into a cleared triangle and as the finished matrix: the same bits; into a filled one: the sum, one rounding each."""
    from acoular_b200 import device as D
    N = 128
    x = torch.randn((K + 1) * N // 2, M, dtype=torch.float32, device='cuda')
    args = (x, N, 'Hanning', '50%', precision)
    up, n = D.csm_upper_accumulate(*args)
    assert n == K
    assert torch.equal(D.csm_finished(*args, 1.0), D.csm_finalize(up, 1.0))
    fill = torch.randn(up.shape, dtype=torch.complex128, device='cuda').triu()
    fill.diagonal(dim1=1, dim2=2).imag.zero_()
    twice, _ = D.csm_upper_accumulate(*args, csm_upper=fill.clone())
    assert torch.equal(twice, fill + up)
