"""Point-spread functions at the edges of their tiles (32 points x 32 sources, 32 mics per chunk), with the sources the
grid in order (a tile right of the diagonal gives its mirror image too), the grid permuted in places, and subsets;
against the oracle, 1e-10 of max."""

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device='cuda')


@pytest.mark.parametrize('G,M', [(1, 3), (31, 31), (32, 32), (33, 33), (64, 5), (65, 64), (97, 65), (160, 20)])
@pytest.mark.parametrize('steer', ['classic', 'inverse', 'true level', 'true location'])
def test_psf_tiles(G, M, steer):
    from acoular_b200 import device as D
    r = np.random.RandomState(G + M)
    mpos = np.vstack([r.uniform(-0.5, 0.5, (2, M)), np.zeros(M)])
    gpos = np.vstack([r.uniform(-0.6, 0.6, (2, G)), np.full(G, 0.7)])
    r0, rm = O.apparent_r(gpos), O.apparent_r(gpos, mpos)
    k = 95.0
    ref = O.psf(steer, r0, rm, k, np.arange(G))
    moved = np.arange(G)
    moved[G // 2:G // 2 + 3] = moved[G // 2:G // 2 + 3][::-1]
    for src in (np.arange(G), moved, np.arange(G)[::-1].copy(), np.arange(0, G, 3)):
        got = D.psf_f64(_dev(r0), _dev(rm), k, _dev(src), steer).cpu().numpy()
        assert np.abs(got - ref[:, src]).max() <= 1e-10 * np.abs(ref).max()
