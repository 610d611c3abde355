"""Windowed transforms: every size of the one-CTA path and every count of mics per CTA, and any range of bins."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('N', [16, 32, 64, 128, 512, 2048, 4096, 8192, 16384])
@pytest.mark.parametrize('M', [1, 3, 6, 9, 33])
def test_spectra_and_bin_ranges(N, M):
    """Against numpy's transform: each of the two FP64 transforms leaves the spectrum of a window within
    4 log2(N) eps sqrt(N) |x|_2 (2-norm), so a product of two within 16 log2(N) eps N |x_i| |x_j|, summed over the
    two windows.  A range of bins has the bits of the whole."""
    from acoular_b200 import device as D
    x = np.random.RandomState(N + M).randn(2 * N, M)
    H = N // 2
    d = torch.as_tensor(x, device='cuda')
    up, n = D.csm_upper_accumulate(d, N, 'Rectangular', 'None', 'complex128')
    assert n == 2
    got = up.cpu().numpy()
    X = np.fft.rfft(x.reshape(2, N, M), axis=1)
    ref = np.einsum('wfi,wfj->fij', X.conj(), X)
    norm = np.linalg.norm(x.reshape(2, N, M), axis=1)
    tol = 16 * np.log2(N) * 2.0**-52 * N * np.einsum('wi,wj->ij', norm, norm)
    err = np.minimum(np.abs(got - ref), np.abs(got - ref.conj()))   # either convention of the conjugate
    i, j = np.triu_indices(M)
    assert (err[:, i, j] <= tol[i, j]).all()
    for lo, nb in ((0, 1), (H, 1), (H // 2, 1), (1, H - 1), (H // 2 - 1, 3), (3, 2), (H // 2 + 1, H // 2), (0, H)):
        part, _ = D.csm_upper_accumulate(d, N, 'Rectangular', 'None', 'complex128', bin_lo=lo, num_bins=nb)
        assert np.array_equal(part.cpu().numpy(), got[lo:lo + nb]), (lo, nb)
