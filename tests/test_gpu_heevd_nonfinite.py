"""Eigendecomposition of a batch with non-finite matrices: a NaN matrix is reported by info (an infinite diagonal entry may
count as converged: what stands beside it is negligible), and the other matrices are as without them."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('bad', [float('nan'), float('inf')])
@pytest.mark.parametrize('M', [2, 5, 33, 64])
def test_non_finite_matrices(M, bad):
    from acoular_b200 import device as D
    x = torch.randn(5, M, M + 2, dtype=torch.complex128, device='cuda')
    c = x @ x.mH
    want, wvec, winfo = D.heevd_f64(c)
    assert not winfo.any()
    for a, b in ((0, 0), (M - 1, 0), (M - 1, M - 1)):
        d = c.clone()
        d[1, a, b] = d[1, b, a] = complex(bad, 0.0)
        d[3] = float('nan')
        ev, vec, info = D.heevd_f64(d)
        assert info[[0, 2, 4]].tolist() == [0, 0, 0] and int(info[3]) == 1
        assert bad == float('inf') or int(info[1]) == 1, (a, b)
        assert torch.isnan(ev[3]).all()
        for i in (0, 2, 4):
            assert torch.equal(ev[i], want[i]) and torch.equal(vec[i], wvec[i])
