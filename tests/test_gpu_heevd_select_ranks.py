"""Selected eigenpairs asked for together: each has the bits of the same one asked for alone."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('M', [4, 33, 150, 257, 700])
def test_ranks_together_and_alone(M):
    from acoular_b200 import device as D
    x = torch.randn(5, M, M + 3, dtype=torch.complex128, device='cuda')
    c = x @ x.mH
    for ranks in ([0, M - 1], [0, 1, M - 1], [0, 1, M - 2, M - 1]):
        lam, vec = D.heevd_select_f64(c, ranks)
        for j, r in enumerate(ranks):
            one, ovec = D.heevd_select_f64(c, [r])
            assert torch.equal(lam[:, j], one[:, 0]) and torch.equal(vec[:, :, j], ovec[:, :, 0])
