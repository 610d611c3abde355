"""The conjugate convention of the cross-spectral matrix, entry by entry: C[i][j] = sum over windows of X_i conj(X_j)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['complex128', 'complex64'])
@pytest.mark.parametrize('N', [16, 64, 512, 2048, 16384])
@pytest.mark.parametrize('M', [2, 9, 33])
def test_sign_of_the_imaginary_part(N, M, precision):
    """Against numpy's transform.  Each of the two FP64 transforms leaves the spectrum of a window within
    4 log2(N) eps sqrt(N) |x|_2 (2-norm), so a product of two within 16 log2(N) eps N |x_i| |x_j|, summed over the two
    windows; complex64 adds the rounding of the spectra and of the sums, at most 16 2^-24 sum |X_i| |X_j|."""
    from acoular_b200 import device as D
    x = np.random.RandomState(3 * N + M).randn(2 * N, M)
    up, n = D.csm_upper_accumulate(torch.as_tensor(x, device='cuda'), N, 'Rectangular', 'None', precision)
    assert n == 2
    X = np.fft.rfft(x.reshape(2, N, M), axis=1)
    ref = np.einsum('wfi,wfj->fij', X, X.conj())
    norm = np.linalg.norm(x.reshape(2, N, M), axis=1)
    tol = np.broadcast_to(16 * np.log2(N) * 2.0**-52 * N * np.einsum('wi,wj->ij', norm, norm), ref.shape)
    if precision == 'complex64':
        tol = tol + 16 * 2.0**-24 * np.einsum('wfi,wfj->fij', np.abs(X), np.abs(X))
    i, j = np.triu_indices(M)
    assert (np.abs(up.cpu().numpy() - ref)[:, i, j] <= tol[:, i, j]).all()
    # the whole matrix, both triangles, of two scaled windows
    full = D.csm_finished(torch.as_tensor(x, device='cuda'), N, 'Rectangular', 'None', precision, 0.5).cpu().numpy()
    assert (np.abs(full - 0.5 * ref) <= tol).all()
