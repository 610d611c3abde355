"""Several host threads, each with a size of its own: a call's launch does not depend on what the other threads call."""

import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _csm(M, B=2):
    x = torch.randn(B, M, 2 * M, dtype=torch.complex128, device='cuda')
    return (x @ x.mH).div_(2 * M)


def _geometry(M, G):
    mpos = torch.rand(3, M, dtype=torch.float64, device='cuda')
    mpos[2] = 0.0
    gpos = torch.rand(3, G, dtype=torch.float64, device='cuda')
    gpos[2] = 0.9
    return mpos, gpos


def _wave_numbers(B=2):
    return torch.linspace(20.0, 40.0, B, dtype=torch.float64, device='cuda')


def _spectra(M):
    from acoular_b200 import device as D
    x = torch.randn(2048, M, dtype=torch.float64, device='cuda')
    return lambda: D.calc_csm(x, 256, 'Hanning', '50%')


def _map(M):
    from acoular_b200 import device as D
    c, k, (mpos, gpos) = _csm(M), _wave_numbers(), _geometry(M, 48)
    return lambda: D.map_f64(c, k, mpos, gpos, 'true level', True, 1.0)


def _map_eig(M):
    from acoular_b200 import device as D
    ev, vec = torch.linalg.eigh(_csm(M))
    ev, vec = ev[:, -8:].contiguous(), vec[:, :, -8:].contiguous()
    k, (mpos, gpos) = _wave_numbers(), _geometry(M, 48)
    return lambda: D.map_eig_f64(ev, vec, k, mpos, gpos, 'true level', True, 1.0)


def _cleansc(M):
    from acoular_b200 import device as D
    c, k, (mpos, gpos) = _csm(M), _wave_numbers(), _geometry(M, 60)
    return lambda: D.cleansc_f64(c.clone(), k, 'true level', True, 1.0, 3, 0.6, 3, mpos=mpos, gpos=gpos, ref=0.0)


def _eigh(M):
    from acoular_b200 import device as D
    c = _csm(M)
    return lambda: D.heevd_f64(c)[0]


def _eigh_select(M):
    from acoular_b200 import device as D
    c = _csm(M)
    return lambda: D.heevd_select_f64(c, [-1])[0]


def _damas(G):
    from acoular_b200 import device as D
    A = torch.rand(2, G, G, dtype=torch.float64, device='cuda').div_(G)
    A.diagonal(dim1=1, dim2=2).fill_(1.0)
    y = torch.rand(2, G, dtype=torch.float64, device='cuda')
    return lambda: D.damas_gauss_seidel(A, y, 1, 1.0, cta_per_bin=4)


@pytest.mark.parametrize('make,sizes', [(_spectra, (3, 40)), (_map, (20, 250)), (_map_eig, (20, 250)),
                                        (_cleansc, (16, 112)), (_cleansc, (120, 200)), (_eigh, (50, 95)),
                                        (_eigh_select, (50, 95)), (_damas, (200, 2000))])
def test_threads_with_different_sizes(make, sizes):
    """Every call of every thread succeeds with the bits of a call alone."""
    calls = [make(n) for n in sizes] * 2
    want = [f() for f in calls]
    torch.cuda.synchronize()
    start, errors, wrong = threading.Barrier(len(calls)), [], []

    def work(i):
        start.wait()
        with torch.cuda.stream(torch.cuda.Stream()):
            got = []
            try:
                for _ in range(200):
                    got.append(calls[i]())
            except RuntimeError as e:
                errors.append(f'size {sizes[i % 2]}: {e}')
            torch.cuda.current_stream().synchronize()
            wrong.extend(i for g in got if not torch.equal(g, want[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert not wrong
