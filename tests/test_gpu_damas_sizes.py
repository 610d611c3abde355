"""DAMAS sweeps at the edges of the two-blocks-ahead form: its smallest grid (more than five blocks of 32 rows), short last
blocks, slices of one and several groups of eight column blocks, empty slices, both cluster sizes and more bins than
clusters resident at once, against the oracle (1e-10 of max, the kernel's bar)."""

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('G,B,cta,n_iter', [(160, 2, 8, 5), (161, 2, 8, 5), (161, 2, 4, 5), (192, 1, 8, 1), (223, 3, 4, 7),
                                            (225, 3, 8, 7), (300, 20, 0, 4), (300, 40, 4, 4), (1000, 2, 8, 3),
                                            (1793, 1, 8, 2), (2500, 1, 4, 2)])
def test_damas_ahead_sizes(G, B, cta, n_iter):
    from acoular_b200 import device as D
    r = np.random.default_rng(G + B)
    A = r.uniform(0.0, 1.0, (B, G, G)) / G
    A[:, np.arange(G), np.arange(G)] = 1.0
    y = r.uniform(-0.2, 1.0, (B, G))
    x0 = r.uniform(0.0, 1.0, (B, G))
    for relax in (1.0, 0.85):
        ref = O.damas_gauss_seidel(A, y, n_iter, relax, x0.copy())
        got = D.damas_gauss_seidel(torch.as_tensor(A, device='cuda'), torch.as_tensor(y, device='cuda'), n_iter, relax,
                                   solution=torch.as_tensor(x0, device='cuda'), cta_per_bin=cta).cpu().numpy()
        assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()
        assert (got >= 0).all()
