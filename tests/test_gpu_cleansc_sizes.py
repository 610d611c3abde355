"""CLEAN-SC at the edges of the cluster form (112 mics, 2048 points for one value per thread, 8192 for four, 15 bins for
the wide variant) and just past them, against the oracle: the same peaks, 1e-5 of max (a float32 result); a bin gives the
same bits alone and among many."""

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device='cuda')


@pytest.mark.parametrize('M,G,B,steer,stopn', [(2, 1, 1, 'classic', 3), (33, 2048, 2, 'true level', 3),
                                               (64, 2049, 1, 'inverse', 2), (65, 300, 16, 'true location', 3),
                                               (112, 777, 2, 'true level', 1), (113, 300, 2, 'true level', 3),
                                               (20, 8192, 2, 'classic', 63), (20, 8193, 1, 'classic', 64),
                                               (31, 2500, 17, 'true level', 4)])
def test_cleansc_sizes(M, G, B, steer, stopn):
    from acoular_b200 import device as D
    r = np.random.RandomState(M + G)
    mpos = np.vstack([r.uniform(-0.5, 0.5, (2, M)), np.zeros(M)])
    gpos = np.vstack([r.uniform(-0.6, 0.6, (2, G)), np.full(G, 0.8)])
    x = r.randn(B, M, 3 * M) + 1j * r.randn(B, M, 3 * M)
    freqs = r.uniform(1500, 6000, B)
    r0, rm = O.apparent_r(gpos), O.apparent_r(gpos, mpos)
    for b in range(B):   # two sources above the noise
        for s, amp in zip(r.randint(0, G, 2), (8.0, 3.0)):
            d = np.linalg.norm(mpos - gpos[:, s:s + 1], axis=0)
            x[b] += amp * np.exp(-2j * np.pi * freqs[b] / 343.0 * d)[:, None] / d[:, None] * r.randn(3 * M)
    csm = x @ x.conj().transpose(0, 2, 1) / (3 * M)
    norm = O.sig_loss_norm(True, M)
    ref = O.beamformer_cleansc_calc(csm, freqs, np.arange(min(B, 2)), r0, rm, 343.0, steer, True, 8, 0.6, stopn)
    k = 2 * np.pi * freqs / 343.0
    geo = dict(mpos=_dev(mpos), gpos=_dev(gpos), ref=0.0)
    got = D.cleansc_f64(_dev(csm), _dev(k), steer, True, norm, 8, 0.6, stopn, **geo).double().cpu().numpy()
    for b in range(min(B, 2)):
        assert np.array_equal(got[b] != 0, ref[b] != 0)
        assert np.abs(got[b] - ref[b]).max() <= 1e-5 * np.abs(ref[b]).max()
    one = D.cleansc_f64(_dev(csm[B - 1:]), _dev(k[B - 1:]), steer, True, norm, 8, 0.6, stopn, **geo)
    assert np.array_equal(one[0].double().cpu().numpy(), got[B - 1])
