"""The FP64 maps at the edges of their tiles (16 grid points, groups of 16 rows, 4-column steps, four or eight warps,
one tile of mics up to 768 and pairs of 384-mic tiles above) and the short cuts of the sincos table lookup.

Bar 1e-10 of the bin's maximum against the oracle, the plain form's; the lookup's short cuts change no bit.
"""

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

STEERS = ['classic', 'inverse', 'true level', 'true location']
TOL = 1e-10


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


def _rel(got, ref):
    got, ref = np.asarray(got), np.asarray(ref)
    return float((np.abs(got - ref).max(-1) / np.abs(ref).max(-1)).max())


@pytest.mark.parametrize('M,G', [(2, 1), (15, 16), (16, 17), (17, 33), (31, 15), (33, 16), (64, 47), (65, 1), (255, 17),
                                 (256, 33), (257, 16), (384, 5), (385, 17), (768, 16), (769, 17), (1100, 9)])
def test_full_csm_map_tiles(M, G):
    from acoular_b200 import device as D
    B = 2
    mpos, gpos, csm, k, r0, rm = _scene(M, G, B, M * 100 + G)
    for i, steer in enumerate(STEERS):
        r_diag = (i + M) % 2 == 0
        norm = O.sig_loss_norm(r_diag, M)
        ref = [O.beamformer_freq(steer, r_diag, norm, r0, rm, k[b], csm[b])[0] for b in range(B)]
        got = D.map_f64(_dev(csm), _dev(k), _dev(mpos), _dev(gpos), steer, r_diag, norm, clip_negative=False)
        assert _rel(got.cpu(), ref) <= TOL, steer
        got = D.map_rm_f64(_dev(csm), _dev(k), _dev(r0), _dev(rm), steer, r_diag, norm, clip_negative=False)
        assert _rel(got.cpu(), ref) <= TOL, steer
    r = np.random.RandomState(7)
    h = r.randn(B, G, M) + 1j * r.randn(B, G, M)
    ref = [O.beamformer_freq_custom(False, 1.0, h[b], csm=csm[b])[0] for b in range(B)]
    assert _rel(D.map_custom_f64(_dev(csm), _dev(h), False, 1.0).cpu(), ref) <= TOL


@pytest.mark.parametrize('M,G,E,B', [(8, 17, 1, 1), (20, 16, 4, 3), (20, 33, 5, 2), (17, 15, 16, 2), (33, 16, 17, 1),
                                     (70, 31, 64, 1), (70, 16, 65, 2), (300, 17, 130, 1), (800, 3, 20, 1)])
def test_eigenvalue_map_tiles(M, G, E, B):
    from acoular_b200 import device as D
    mpos, gpos, csm, k, r0, rm = _scene(M, G, B, M * 100 + E)
    ev, vec = np.linalg.eigh(csm)
    ev, vec = np.ascontiguousarray(ev[:, -E:]), np.ascontiguousarray(vec[:, :, -E:])
    for i, steer in enumerate(STEERS):
        r_diag = i % 2 == 0
        ref = [O.beamformer_freq_eig(steer, r_diag, 1.0, r0, rm, k[b], ev[b], vec[b])[0] for b in range(B)]
        got = D.map_eig_f64(_dev(ev), _dev(vec), _dev(k), _dev(mpos), _dev(gpos), steer, r_diag, 1.0,
                            clip_negative=False)
        assert _rel(got.cpu(), ref) <= TOL, steer
        got = torch.stack([D.map_eig_rm_f64(_dev(ev[b:b + 1]), _dev(vec[b:b + 1]), k[b], _dev(r0), _dev(rm), steer,
                                            r_diag, 1.0) for b in range(B)])
        assert _rel(got.cpu(), ref) <= TOL, steer


@pytest.mark.parametrize('B', [1, 3, 4, 5, 7])
def test_one_component_several_bins_per_thread(B):
    """One component on a grid large enough for four bins per thread: each bin equals the same bin alone."""
    from acoular_b200 import device as D
    M, G = 3, 128 * 8 * 148 + 5
    mpos, gpos, csm, k, r0, rm = _scene(M, G, B, B)
    ev, vec = np.linalg.eigh(csm)
    ev, vec = np.ascontiguousarray(ev[:, -1:]), np.ascontiguousarray(vec[:, :, -1:])
    geo = (_dev(mpos), _dev(gpos))
    got = D.map_eig_f64(_dev(ev), _dev(vec), _dev(k), *geo, 'true level', True, 1.5, clip_negative=False).cpu().numpy()
    ref = [O.beamformer_freq_eig('true level', True, 1.5, r0, rm, k[b], ev[b], vec[b])[0] for b in range(B)]
    assert _rel(got, ref) <= TOL
    one = [D.map_eig_f64(_dev(ev[b:b + 1]), _dev(vec[b:b + 1]), _dev(k[b:b + 1]), geo[0], geo[1][:, :70].contiguous(),
                         'true level', True, 1.5, clip_negative=False).cpu().numpy()[0] for b in range(B)]
    assert np.array_equal(got[:, :70], np.stack(one))


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
