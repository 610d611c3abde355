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


@pytest.mark.parametrize('N', [16, 64, 512, 2048, 16384])
@pytest.mark.parametrize('M', [2, 9, 33])
def test_complex64_spectra(N, M):
    """Spectra rounded to FP32 (2^-24 each component, so 2^-23 of |X_i| |X_j| for a product of two, with a factor of 2
    for real and imaginary parts) and summed over two windows in FP32 (four FMAs per component, at most 2^-24 of
    2 sum |X_i| |X_j| each): within 16 2^-24 sum |X_i| |X_j|; the FP64 transforms' own error as above."""
    from acoular_b200 import device as D
    x = np.random.RandomState(N + M + 1).randn(2 * N, M).astype(np.float32)
    up, _ = D.csm_upper_accumulate(torch.as_tensor(x, device='cuda'), N, 'Rectangular', 'None', 'complex64')
    X = np.fft.rfft(x.astype(np.float64).reshape(2, N, M), axis=1)
    ref = np.einsum('wfi,wfj->fij', X.conj(), X)
    size = np.einsum('wfi,wfj->fij', np.abs(X), np.abs(X))
    norm = np.linalg.norm(x.astype(np.float64).reshape(2, N, M), axis=1)
    tol = 16 * 2.0**-24 * size + 16 * np.log2(N) * 2.0**-52 * N * np.einsum('wi,wj->ij', norm, norm)
    got = up.cpu().numpy()
    err = np.minimum(np.abs(got - ref), np.abs(got - ref.conj()))
    i, j = np.triu_indices(M)
    assert (err[:, i, j] <= tol[:, i, j]).all()
