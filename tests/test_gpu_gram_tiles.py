"""The Welch Gram at the edges of its tiles (complex128: 32 mics, complex64: 64, 16 windows per stage): the accumulation
is the reference's chain of two FMAs per window and component, so equality is bit for bit, and the matrix written
finished has the bits of the accumulated and finalised one."""

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype', [np.complex128, np.complex64])
@pytest.mark.parametrize('M', [1, 2, 7, 16, 17, 31, 32, 33, 48, 64, 65, 97, 113, 130])
def test_calc_csm_bits(M, dtype):
    from acoular_b200 import fastFuncs as F
    r = np.random.RandomState(M)
    ref = np.triu(r.randn(3, M, M) + 1j * r.randn(3, M, M)).astype(dtype)
    got = ref.copy()
    for _ in range(3):
        spec = (r.randn(3, M) + 1j * r.randn(3, M)).astype(dtype)
        O.calc_csm_upper(ref, spec)
        F.calcCSM(got, spec)
    assert np.array_equal(got, ref)


@pytest.mark.parametrize('precision', ['complex128', 'complex64'])
@pytest.mark.parametrize('M,K', [(1, 1), (33, 2), (40, 15), (40, 16), (40, 17), (64, 31), (65, 33), (20, 100)])
def test_windows_at_once_equal_one_by_one(M, K, precision):
    from acoular_b200 import device as D
    N = 64
    x = torch.as_tensor(np.random.RandomState(M + K).randn(N // 2 * (K + 1), M), device='cuda')
    full, n = D.csm_upper_accumulate(x, N, 'Hanning', '50%', precision)
    assert n == K
    one = torch.zeros_like(full)
    for w in range(K):
        D.csm_upper_accumulate(x, N, 'Hanning', '50%', precision, csm_upper=one, first_window=w, windows=1)
    assert torch.equal(full, one)


@pytest.mark.parametrize('precision', ['complex128', 'complex64', 'tc_tf32', 'tc_bf16x3'])
@pytest.mark.parametrize('M,K', [(1, 1), (2, 40), (33, 17), (64, 16), (65, 33), (113, 9), (130, 3)])
def test_finished_matrix_bits(M, K, precision):
    from acoular_b200 import device as D
    N, scale = 128, 0.37
    x = torch.as_tensor(np.random.RandomState(M * K).randn(N // 4 * (K + 3) + 5, M).astype('f4'), device='cuda')
    up, n = D.csm_upper_accumulate(x, N, 'Hamming', '75%', precision, bin_lo=3, num_bins=40)
    assert n == K
    ref = D.csm_finalize(up, scale)
    got = D.csm_finished(x, N, 'Hamming', '75%', precision, scale, bin_lo=3, num_bins=40)
    assert torch.equal(got, ref)
    if precision.startswith('complex'):   # several chunks: the accumulating route
        small = M * 40 * 16 * max(1, K // 3)
        assert torch.equal(D.csm_finished(x, N, 'Hamming', '75%', precision, scale, bin_lo=3, num_bins=40,
                                          max_workspace_bytes=small), ref)
    # no complete window: the accumulating route's zeros times the scale
    none = D.csm_finished(x[:N - 1], N, 'Hamming', '75%', precision, scale)
    assert not none.any()
