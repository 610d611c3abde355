"""The bounded waits between the CTAs of a cluster: where one runs out the result is marked, never a plausible number.

Limits of 100 ns, far shorter than the steps that the waits cover, and of a few microseconds, about what they take: waits
run out on a normal input (no fault, no trap, nothing that never finishes), early and late, and in any CTA of a cluster.
"""

import contextlib

import pytest
import torch

pytestmark = pytest.mark.gpu

LIMITS = [100, 100, 2000, 3000, 5000, 8000]


@contextlib.contextmanager
def short_waits(ns):
    from acoular_b200 import _native as N
    prev = N.lib().acb_tc_set_wait_limit_ns(ns)
    try:
        yield
    finally:
        torch.cuda.synchronize()
        N.lib().acb_tc_set_wait_limit_ns(prev)


@pytest.mark.parametrize('G,cta', [(161, 4), (500, 4), (500, 8), (4000, 4)])
def test_damas_marks_the_bin(G, cta):
    """Each bin is the full run's, bit for bit, or NaN throughout."""
    from acoular_b200 import device as D
    B = 3
    A = torch.rand(B, G, G, dtype=torch.float64, device='cuda').div_(G)
    A.diagonal(dim1=1, dim2=2).fill_(1.0)
    y = torch.rand(B, G, dtype=torch.float64, device='cuda')
    full = D.damas_gauss_seidel(A, y, 6, 1.0, cta_per_bin=cta)
    assert torch.isfinite(full).all()
    marked = 0
    for ns in LIMITS:
        with short_waits(ns):
            got = D.damas_gauss_seidel(A, y, 6, 1.0, cta_per_bin=cta)
        for b in range(B):
            bad = torch.isnan(got[b])
            assert bad.all() or torch.equal(got[b], full[b])
            marked += int(bad.all())
    assert marked > 0
    assert torch.equal(D.damas_gauss_seidel(A, y, 6, 1.0, cta_per_bin=cta), full)   # and the device is as before


@pytest.mark.parametrize('M', [100, 180, 256, 330])
def test_eigendecomposition_marks_the_matrix(M):
    """Clusters of 1, 2, 4 and 8 CTAs.  Each matrix is the full run's, bit for bit, or NaN, with info 1."""
    from acoular_b200 import device as D
    B = 12
    x = torch.randn(B, M, M + 5, dtype=torch.complex128, device='cuda')
    c = x @ x.mH
    ev, vec, info = D.heevd_f64(c)
    lam, sel = D.heevd_select_f64(c, [0, -1])
    assert not info.any()
    marked = 0
    for ns in LIMITS:
        with short_waits(ns):
            e2, v2, i2 = D.heevd_f64(c)
            l2, s2 = D.heevd_select_f64(c, [0, -1])
        for b in range(B):
            if int(i2[b]):
                assert torch.isnan(e2[b]).all() and torch.isnan(v2[b]).all()
            else:
                assert torch.equal(e2[b], ev[b]) and torch.equal(v2[b], vec[b])
            bad = torch.isnan(l2[b])
            if bad.any():
                assert bad.all() and torch.isnan(s2[b]).all()
            else:
                assert torch.equal(l2[b], lam[b]) and torch.equal(s2[b], sel[b])
            marked += int(i2[b]) + int(bad.all())
    assert marked > 0
    assert torch.equal(D.heevd_f64(c)[0], ev)   # and the device is as before


def test_selected_pairs_of_nan_matrices():
    """NaN in, NaN out; the other matrices are as without them."""
    from acoular_b200 import device as D
    for M in (5, 64, 300, 600):
        x = torch.randn(4, M, M + 2, dtype=torch.complex128, device='cuda')
        c = x @ x.mH
        want, wvec = D.heevd_select_f64(c, [0, -1])
        c[1, M - 1, M - 1] = float('nan')
        c[2] = float('nan')
        lam, vec = D.heevd_select_f64(c, [0, -1])
        for b in (0, 3):
            assert torch.equal(lam[b], want[b]) and torch.equal(vec[b], wvec[b])
        for b in (1, 2):
            assert torch.isnan(lam[b]).all() and torch.isnan(vec[b]).all()
