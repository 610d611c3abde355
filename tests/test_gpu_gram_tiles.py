"""The complex128 Welch Gram at the edges of its tiles (32 mics, 16 windows per stage): the accumulation is the
reference's chain of two FMAs per window and component, so equality is bit for bit."""

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('M', [1, 2, 7, 16, 17, 31, 32, 33, 48, 64, 65, 97, 130])
def test_calc_csm_bits(M):
    from acoular_b200 import fastFuncs as F
    r = np.random.RandomState(M)
    ref = np.triu(r.randn(3, M, M) + 1j * r.randn(3, M, M))
    got = ref.copy()
    for _ in range(3):
        spec = r.randn(3, M) + 1j * r.randn(3, M)
        O.calc_csm_upper(ref, spec)
        F.calcCSM(got, spec)
    assert np.array_equal(got, ref)


@pytest.mark.parametrize('M,K', [(1, 1), (33, 2), (40, 15), (40, 16), (40, 17), (64, 31), (65, 33), (20, 100)])
def test_windows_at_once_equal_one_by_one(M, K):
    from acoular_b200 import device as D
    N = 64
    x = torch.as_tensor(np.random.RandomState(M + K).randn(N // 2 * (K + 1), M), device='cuda')
    full, n = D.csm_upper_accumulate(x, N, 'Hanning', '50%')
    assert n == K
    one = torch.zeros_like(full)
    for w in range(K):
        D.csm_upper_accumulate(x, N, 'Hanning', '50%', csm_upper=one, first_window=w, windows=1)
    assert torch.equal(full, one)
