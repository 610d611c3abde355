"""The QL rotations outside the range of the plain sum of squares: matrices of very small and very large norm."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('scale', [1e-145, 1e-142, 1.0, 1e142, 1e145])
@pytest.mark.parametrize('M', [2, 31, 64, 112])
def test_scaled_matrices(M, scale):
    """Bars of the other eigendecomposition tests: 1e-12 of the largest eigenvalue."""
    from acoular_b200 import device as D
    r = np.random.RandomState(M)
    x = r.randn(3, M, M + 9) + 1j * r.randn(3, M, M + 9)
    a = x @ x.conj().transpose(0, 2, 1) / M
    w, v, info = D.heevd_f64(torch.as_tensor(a * scale, device='cuda'))
    w, v = w.cpu().numpy() / scale, v.cpu().numpy()
    assert not int(info.max())
    ref = np.linalg.eigvalsh(a)
    assert np.abs(w - ref).max() <= 1e-12 * ref.max()
    assert np.abs(a @ v - v * w[:, None, :]).max() <= 1e-12 * ref.max()
    assert np.abs(v.conj().transpose(0, 2, 1) @ v - np.eye(M)).max() <= 1e-12
