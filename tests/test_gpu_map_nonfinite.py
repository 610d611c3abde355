"""FP64 maps of a CSM with non-finite entries: what diagonal removal takes out may be anything, the rest counts as it is."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# below, at and above whole groups of 4 columns, 8 and 16 rows; one tile, eight warps, pairs of tiles
MICS = [2, 3, 7, 8, 9, 15, 16, 17, 30, 61, 64, 255, 257, 300, 770]


def _inputs(M, B=2, G=37):
    rng = np.random.RandomState(M)
    x = rng.randn(B, M, M + 3) + 1j * rng.randn(B, M, M + 3)
    csm = torch.as_tensor(x @ x.conj().transpose(0, 2, 1) / M, device='cuda')
    mpos = torch.as_tensor(rng.uniform(-0.3, 0.3, (3, M)), device='cuda')
    gpos = torch.as_tensor(np.vstack([rng.uniform(-0.4, 0.4, (2, G)), np.full((1, G), 1.1)]), device='cuda')
    k = torch.tensor([31.0, 95.0], dtype=torch.float64, device='cuda')
    rm = torch.linalg.vector_norm(gpos[:, :, None] - mpos[:, None, :], dim=0).contiguous()
    r0 = torch.linalg.vector_norm(gpos, dim=0)
    steer = torch.as_tensor(rng.randn(B, G, M) + 1j * rng.randn(B, G, M), device='cuda')
    return csm, k, mpos, gpos, r0, rm, steer


def _maps(D, csm, k, mpos, gpos, r0, rm, steer, r_diag):
    yield 'positions', D.map_f64(csm, k, mpos, gpos, 'true level', r_diag, 1.0, clip_negative=False)
    yield 'distances', D.map_rm_f64(csm, k, r0, rm, 'inverse', r_diag, 1.0, clip_negative=False)
    yield 'custom', D.map_custom_f64(csm, steer, r_diag, 1.0)


@pytest.mark.parametrize('bad', [float('nan'), float('inf'), float('-inf')])
@pytest.mark.parametrize('M', MICS)
def test_removed_diagonal_may_be_anything(M, bad):
    """The same bits as with a finite diagonal: all mics, the first, the last, one in between (no tolerance: the entries
    take no part)."""
    from acoular_b200 import device as D
    csm, *rest = _inputs(M)
    want = dict(_maps(D, csm, *rest, True))
    assert all(torch.isfinite(w).all() for w in want.values())
    for mics in (range(M), [0], [M - 1], [M // 2]):
        c = csm.clone()
        for m in mics:
            c[:, m, m] = complex(bad, 0.0)
        for name, got in _maps(D, c, *rest, True):
            assert torch.equal(got, want[name]), (name, mics)


@pytest.mark.parametrize('M', MICS)
def test_kept_infinite_diagonal(M):
    """A kept diagonal enters as a positive square times its entry: infinite, and not a number nowhere."""
    from acoular_b200 import device as D
    csm, *rest = _inputs(M)
    for m in (0, M // 2, M - 1):
        c = csm.clone()
        c[:, m, m] = complex(float('inf'), 0.0)
        for name, got in _maps(D, c, *rest, False):
            assert (got == float('inf')).all(), (name, m)


@pytest.mark.parametrize('M', MICS)
def test_infinite_entry_off_the_diagonal(M):
    """C_ab = inf enters as Re(conj(h_a) inf h_b) = inf (sign(h_a h_b) of the real parts + of the imaginary parts): an
    infinity of that sign where the two agree, else not a number; nothing that does not count adds to it."""
    from acoular_b200 import device as D
    csm, *_, steer = _inputs(M)
    for a, b in ((0, M - 1), (M - 2, M - 1), (0, 1), (M // 2 - 1, M // 2)):
        if a < 0 or a == b:
            continue
        c = csm.clone()
        c[:, a, b] = c[:, b, a] = complex(float('inf'), 0.0)
        got = D.map_custom_f64(c, steer, True, 1.0)
        s = [torch.sign(steer[:, :, a].real) * torch.sign(steer[:, :, b].real),
             torch.sign(steer[:, :, a].imag) * torch.sign(steer[:, :, b].imag)]
        same = s[0] == s[1]
        assert torch.equal(got[same], s[0][same] * float('inf')), (a, b)
        assert torch.isnan(got[~same]).all(), (a, b)
