"""Point-spread functions of some of the grid's points: the columns of the full function, bit for bit, in every tile form."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _geometry(M, G, seed):
    r = np.random.RandomState(seed)
    mpos = torch.as_tensor(np.vstack([r.uniform(-0.5, 0.5, (2, M)), np.zeros(M)]), device='cuda')
    gpos = torch.as_tensor(np.vstack([r.uniform(-1, 1, (2, G)), np.full(G, 0.8)]), device='cuda')
    rm = (gpos.T[:, None, :] - mpos.T[None]).norm(dim=2).contiguous()
    return gpos.norm(dim=0), rm


@pytest.mark.parametrize('steer', ['classic', 'inverse', 'true level', 'true location'])
@pytest.mark.parametrize('M,G', [(3, 33), (40, 545), (33, 700)])
def test_subset_equals_columns(M, G, steer):
    """8, 16 or 32 sources per CTA, full and ragged, against all of them in order (mirrored from 545 points on)."""
    from acoular_b200 import device as D
    r0, rm = _geometry(M, G, M + G)
    full = D.psf_f64(r0, rm, 40.0, np.arange(G), steer)
    order = np.random.RandomState(G).permutation(G)
    assert torch.equal(D.psf_f64(r0, rm, 40.0, order, steer), full[:, torch.as_tensor(order, device='cuda')])
    for S in (1, 7, 8, 9, 16, 17, 31, 32, 33):
        if S < G:
            sub = order[:S]
            got = D.psf_f64(r0, rm, 40.0, sub, steer)
            assert torch.equal(got, full[:, torch.as_tensor(sub, device='cuda')]), S


@pytest.mark.parametrize('steer', ['classic', 'inverse', 'true level', 'true location'])
@pytest.mark.parametrize('S', [64, 67, 72, 128, 129])
def test_many_points(S, steer):
    """A grid large enough for 16 and 32 sources per CTA; a source outside the grid gives NaN and no other change."""
    from acoular_b200 import device as D
    M, G = 5, 20003
    r0, rm = _geometry(M, G, S)
    src = np.random.RandomState(S).permutation(G)[:S]
    got = D.psf_f64(r0, rm, 55.0, src, steer)
    for j in (0, 7, 15, 31, 40, S - 1):
        assert torch.equal(got[:, j:j + 1], D.psf_f64(r0, rm, 55.0, src[j:j + 1], steer))
    bad = torch.as_tensor(src, device='cuda')
    bad[S // 2] = G
    out = D.psf_f64(r0, rm, 55.0, bad, steer)
    keep = torch.arange(S, device='cuda') != S // 2
    assert torch.isnan(out[:, S // 2]).all() and torch.equal(out[:, keep], got[:, keep])
