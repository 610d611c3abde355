"""The Grams in their small and large tiles (complex128: 32 x 16 and 32 x 32, complex64: 32 x 32 and 64 x 64): the same
chain of FMAs, so the same bits."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('M', [1, 15, 16, 17, 31, 32, 33, 47, 49, 64, 65, 80, 97, 113, 130])
def test_few_bins_equal_many_bins(M):
    from acoular_b200 import device as D
    N = 1024   # 513 bins: 32 x 32 tiles; a few of them: 32 x 16
    x = torch.as_tensor(np.random.RandomState(M).randn(N // 2 * 38, M), device='cuda')
    many = D.calc_csm(x, N, 'Hanning', '50%', 'complex128')
    up, _ = D.csm_upper_accumulate(x, N, 'Hanning', '50%', 'complex128')
    for lo, nb in ((0, 1), (100, 7), (512, 1)):
        few = D.calc_csm(x, N, 'Hanning', '50%', 'complex128', bin_lo=lo, num_bins=nb)
        assert torch.equal(few, many[lo:lo + nb])
        part, _ = D.csm_upper_accumulate(x, N, 'Hanning', '50%', 'complex128', bin_lo=lo, num_bins=nb)
        assert torch.equal(part, up[lo:lo + nb])


@pytest.mark.parametrize('M', [1, 31, 32, 33, 63, 64, 65, 96, 97, 129])
def test_few_bins_equal_many_bins_c64(M):
    from acoular_b200 import device as D
    N = 1024   # 513 bins: 64 x 64 tiles above 32 mics; a few of them: 32 x 32
    x = torch.as_tensor(np.random.RandomState(M + 1).randn(N // 2 * 38, M), device='cuda', dtype=torch.float32)
    many = D.calc_csm(x, N, 'Hanning', '50%', 'complex64')
    up, _ = D.csm_upper_accumulate(x, N, 'Hanning', '50%', 'complex64')
    for lo, nb in ((0, 1), (100, 7), (512, 1)):
        few = D.calc_csm(x, N, 'Hanning', '50%', 'complex64', bin_lo=lo, num_bins=nb)
        assert torch.equal(few, many[lo:lo + nb])
        part, _ = D.csm_upper_accumulate(x, N, 'Hanning', '50%', 'complex64', bin_lo=lo, num_bins=nb)
        assert torch.equal(part, up[lo:lo + nb])
