"""The short cuts of the sincos table lookup change no bit of the FP64 maps and point-spread functions."""

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device='cuda')


def _scene(M, G, B, seed):
    r = np.random.RandomState(seed)
    mpos = np.vstack([r.uniform(-0.5, 0.5, (2, M)), np.zeros(M)])
    gpos = np.vstack([r.uniform(-0.6, 0.6, (2, G)), np.full(G, 0.8)])
    x = r.randn(B, M, 2 * M + 3) + 1j * r.randn(B, M, 2 * M + 3)
    csm = x @ x.conj().transpose(0, 2, 1) / (2 * M)
    k = r.uniform(5, 300, B)
    return mpos, gpos, csm, k, O.apparent_r(gpos), O.apparent_r(gpos, mpos)


@pytest.mark.parametrize('kmax', [3.0, 150.0, 1400.0])
def test_sincos_lookup_short_cuts_change_no_bit(kmax):
    """A table without its meta entry (no distance limit, no tags) makes every lookup; the results are the same."""
    from acoular_b200 import device as D
    mpos, gpos, csm, k, r0, rm = _scene(48, 5000, 3, 11)
    k = np.array([kmax, 0.7 * kmax, 0.1 * kmax])
    args = (_dev(csm), _dev(k), _dev(mpos), _dev(gpos), 'true level', True, 1.0)
    src = np.arange(0, 5000, 61)
    psf_args = (_dev(r0), _dev(rm), kmax, src, 'inverse')
    got, psf = D.map_f64(*args).cpu(), D.psf_f64(*psf_args).cpu()
    full = D.sincos_table_device('cuda:0')
    key = 0xfffffffe
    slot = (((key * 0x9E3779B97F4A7C15) & (2 ** 64 - 1)) >> 20) & (full.numel() - 1)
    word = int(full[slot])
    assert (word >> 32) & 0xffffffff == key and 0 < word & 0xffff <= 0x8000
    try:
        full[slot] = (0xfffffffd << 32) - (1 << 64)   # a key that no argument has: no meta entry
        assert torch.equal(got, D.map_f64(*args).cpu())
        assert torch.equal(psf, D.psf_f64(*psf_args).cpu())
    finally:
        full[slot] = word
