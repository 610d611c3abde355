"""DAMAS sweeps from a start with NaN or infinite values (a focus point on a microphone gives one): they count for the
rows before them only, as in the row-by-row sweep, and are gone after their own row."""

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('bad', [float('nan'), float('inf')])
@pytest.mark.parametrize('G,cta', [(40, 8), (161, 4), (300, 4), (300, 8), (1000, 8)])
def test_non_finite_start(G, cta, bad):
    """Against the oracle (1e-10 of max, the kernel's bar), at the first, middle and last rows of a block and of the grid."""
    from acoular_b200 import device as D
    r = np.random.default_rng(G)
    A = r.uniform(0.0, 1.0, (1, G, G)) / G
    A[:, np.arange(G), np.arange(G)] = 1.0
    y = r.uniform(0.1, 1.0, (1, G))
    for at in ([0], [5], [31], [G // 2], [G // 2, G // 2 + 3], [G - 1]):
        x0 = y.copy()
        x0[0, at] = bad
        for n_iter in (1, 2, 4):
            ref = O.damas_gauss_seidel(A, y, n_iter, 1.0, x0.copy())
            assert np.isfinite(ref).all()
            got = D.damas_gauss_seidel(torch.as_tensor(A, device='cuda'), torch.as_tensor(y, device='cuda'), n_iter, 1.0,
                                       solution=torch.as_tensor(x0, device='cuda'), cta_per_bin=cta).cpu().numpy()
            assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max(), (at, n_iter)
