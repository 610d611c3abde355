"""CLEAN-SC of many bins: clusters of one to eight CTAs per bin, each bin with the bits of the same bin among a few."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('M,G,B', [(5, 256, 40), (5, 257, 100), (5, 1024, 320), (5, 1025, 320), (64, 60, 310), (64, 2049, 70),
                                   (80, 100, 40), (112, 300, 160), (112, 1025, 80), (20, 4097, 70)])
def test_many_bins(M, G, B):
    from acoular_b200 import device as D
    r = np.random.RandomState(M + G + B)
    mpos = torch.as_tensor(np.vstack([r.uniform(-0.5, 0.5, (2, M)), np.zeros(M)]), device='cuda')
    gpos = torch.as_tensor(np.vstack([r.uniform(-0.6, 0.6, (2, G)), np.full(G, 0.8)]), device='cuda')
    k = torch.as_tensor(r.uniform(30, 110, B), device='cuda')
    x = torch.randn(B, M, 3 * M, dtype=torch.complex128, device='cuda')
    for s, amp in zip(r.randint(0, G, 2), (8.0, 3.0)):
        d = (mpos - gpos[:, s:s + 1]).norm(dim=0)
        x += amp * torch.exp(-1j * k[:, None] * d)[:, :, None] * torch.randn(B, 1, 3 * M, dtype=torch.complex128, device='cuda')
    c = x @ x.mH / (3 * M)
    geo = dict(mpos=mpos, gpos=gpos, ref=0.0)
    got = D.cleansc_f64(c, k, 'true level', True, 1.0, 7, 0.6, 3, **geo)
    few = torch.cat([D.cleansc_f64(c[i:i + 5], k[i:i + 5], 'true level', True, 1.0, 7, 0.6, 3, **geo) for i in range(0, B, 5)])
    assert torch.equal(got, few)
