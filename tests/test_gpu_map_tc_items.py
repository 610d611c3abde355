"""Tensor-core map: every (bin, tile, group) item reaches its place for tile counts around the SM count."""

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['fp16', 'tf32'])
@pytest.mark.parametrize('M,tiles,nb,tuning', [(16, 1, 700, (16, 1)), (16, 147, 5, (16, 1)), (40, 148, 5, (16, 1)),
                                               (16, 149, 9, (16, 1)), (150, 37, 11, (4, 2)), (150, 50, 7, (4, 3)),
                                               (520, 1, 160, (16, 3)), (520, 75, 4, (8, 5))])
def test_items_of_many_bins_equal_single_bins(M, tiles, nb, tuning, precision):
    """A CTA steps through its items by adding the grid's stride; a bin's map alone starts elsewhere, walks
    otherwise and has the same arithmetic, so its bits are the same (no tolerance)."""
    from acoular_b200 import device as D
    dev = torch.device('cuda')
    rng = np.random.RandomState(M + tiles + nb)
    G = 128 * tiles - 5
    mpos = np.vstack([rng.uniform(-0.5, 0.5, (2, M)), np.zeros((1, M))])
    gpos = np.vstack([rng.uniform(-0.4, 0.4, (2, G)), np.full((1, G), -0.6)])
    freqs = np.linspace(1000.0, 9000.0, nb)
    a = rng.randn(nb, M, 3) + 1j * rng.randn(nb, M, 3)
    csm = a @ a.conj().transpose(0, 2, 1) + 0.1 * np.eye(M)
    dc, dk = torch.as_tensor(csm, device=dev), torch.as_tensor(2 * np.pi * freqs / 343.0, device=dev)
    dm, dg = torch.as_tensor(mpos, device=dev), torch.as_tensor(gpos, device=dev)

    def run(sel):
        err = torch.zeros(1, dtype=torch.int32, device=dev)
        out = D.map_tc(dc[sel].contiguous(), dk[sel].contiguous(), dm, dg, 'true location', True,
                       O.sig_loss_norm(True, M), clip_negative=True, precision=precision, tuning=tuning,
                       error_word=err)
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        return out.cpu().numpy()

    full = run(slice(0, nb))
    for b in sorted({0, 1, nb // 2, nb - 2, nb - 1}):
        assert np.array_equal(full[b], run(slice(b, b + 1))[0]), b
