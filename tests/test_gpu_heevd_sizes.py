"""The eigendecomposition at the edges of its size rules: rows per CTA of the cluster form (155, 210, 276, 339 rows in 1,
2, 4, 8 CTAs, the global-memory form above and for many small matrices), and the register rows of the selected columns'
back-transformation.  Bars of the other eigendecomposition tests: 1e-12 of the largest eigenvalue, select 1e-11."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _matrices(B, M):
    r = np.random.RandomState(M)
    x = r.randn(B, M, M + 9) + 1j * r.randn(B, M, M + 9)
    return x @ x.conj().transpose(0, 2, 1) / M


@pytest.mark.parametrize('B,M', [(2, 3), (2, 31), (2, 47), (300, 33), (2, 155), (2, 156), (1, 210), (1, 211), (1, 276),
                                 (1, 277), (1, 339), (1, 340)])
def test_full_decomposition_sizes(B, M):
    from acoular_b200 import device as D
    a = _matrices(B, M)
    w, v, info = D.heevd_f64(torch.as_tensor(a, device='cuda'))
    w, v = w.cpu().numpy(), v.cpu().numpy()
    assert not int(info.max())
    ref = np.linalg.eigvalsh(a)
    assert np.abs(w - ref).max() <= 1e-12 * ref.max()
    assert np.abs(a @ v - v * w[:, None, :]).max() <= 1e-12 * ref.max()
    assert np.abs(v.conj().transpose(0, 2, 1) @ v - np.eye(M)).max() <= 1e-12


@pytest.mark.parametrize('B,M', [(300, 33), (2, 64), (2, 65), (2, 128), (2, 129), (1, 257), (1, 512), (1, 513)])
def test_selected_sizes(B, M):
    from acoular_b200 import device as D
    a = _matrices(B, M)
    ranks = sorted({0, M // 3, M - 1})
    w, v = D.heevd_select_f64(torch.as_tensor(a, device='cuda'), ranks)
    w, v = w.cpu().numpy(), v.cpu().numpy()
    ref = np.linalg.eigvalsh(a)
    assert np.abs(w - ref[:, ranks]).max() <= 1e-12 * ref.max()
    assert np.abs(a @ v - v * w[:, None, :]).max() <= 1e-11 * ref.max()
    assert np.abs(np.linalg.norm(v, axis=1) - 1.0).max() <= 1e-12
