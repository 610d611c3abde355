"""Cases for timing the framework: the calls an acoustic-imaging program makes, over the sizes it meets.

A microphone-array analysis estimates the cross-spectral matrix (CSM) of its channels and maps it onto a grid of
focus points, plainly or with an eigenvalue or deconvolution method.  Every case is one such call, or a short chain of
them, through the public entry points of :mod:`acoular_b200.device` on device-resident data; one case is the whole call
from host samples through the Acoular-compatible classes.  Sizes are those of the workloads in
:mod:`acoular_b200.workloads` (64 microphones with a 41 x 41 grid, 256 microphones with a 401 x 401 grid) and odd ones
between and beyond them.
"""

import math

import numpy as np
import torch

import acoular_b200 as ac
from acoular_b200 import device as D
from acoular_b200.microphones import disk_mics

FS = 51200.0
C0 = 343.0
OVERLAP = {'None': 1, '50%': 2, '75%': 4, '87.5%': 8}
BLOCKS = (128, 256, 512, 1024, 2048, 4096, 8192, 16384)
STEER = ('classic', 'inverse', 'true level', 'true location')


# ------------------------------------------------------------------------------------------------
# cases
# ------------------------------------------------------------------------------------------------
def listed():
    band64 = dict(mics=64, radius=0.25, nx=41, ny=41, nz=1, extent=0.4, z=-0.3, steer='true level', r_diag=True,
                  block=128, bin_lo=18, bins=5)
    plane256 = dict(mics=256, radius=0.5, nx=401, ny=401, nz=1, extent=2.0, z=-1.0, steer='true level', r_diag=True,
                    block=1024)
    return [
        # A quick look at one second of a 64-channel recording held on the device: CSM of all bins and the map of the
        # 8 kHz third-octave band.  The smallest call of an interactive session or of a monitoring loop.
        dict(band64, name='analysis_64ch', kind='analysis', samples=51200, dtype='float64', window='Hanning',
             overlap='50%', precision='complex128'),
        # The same analysis as an Acoular user writes it: host samples into TimeSamples, PowerSpectra, BeamformerBase
        # and synthetic(8000, 3), the band map back on the host.
        dict(band64, name='synthetic_64ch', kind='synthetic', samples=51200, dtype='float64', window='Hanning',
             overlap='50%', precision='complex128'),
        # CSM of ten seconds of a 256-channel array in the reference's precision: the spectral half of a measurement
        # campaign's evaluation.
        dict(name='csm_256ch_c128', kind='csm', mics=256, samples=512000, dtype='float32', block=1024,
             window='Hanning', overlap='50%', precision='complex128'),
        # CSM in single precision with fine frequency resolution, an odd number of channels (some switched off),
        # another window and a larger overlap.
        dict(name='csm_113ch_c64', kind='csm', mics=113, samples=153600, dtype='float32', block=4096,
             window='Blackman', overlap='75%', precision='complex64'),
        # The tensor-core CSM that goes with the tensor-core map on the 256-channel measurement.
        dict(name='csm_256ch_tc', kind='csm', mics=256, samples=512000, dtype='float32', block=1024,
             window='Hanning', overlap='50%', precision='tc_tf32'),
        # Maps of a twelve-bin band on a fine plane grid in the reference's precision: the map half of an evaluation.
        dict(plane256, name='map_256mic_plane', kind='map', form='f64', bin_lo=160, bins=12),
        # A volume in front of a larger array with the reference point off the origin, full CSM, another steering
        # formulation; neither microphones nor grid points fill whole tiles.
        dict(name='map_300mic_box', kind='map', form='f64', mics=300, radius=0.6, nx=31, ny=27, nz=19, extent=1.5,
             z=0.8, steer='true location', r_diag=False, ref=0.1, block=1024, bin_lo=60, bins=6),
        # All 513 bins of the 256-channel measurement on the fine grid with the tensor-core form: the batch evaluation.
        dict(plane256, name='map_256mic_tc', kind='map', form='fp16', bin_lo=0, bins=513),
        # Eigenvalue beamforming with the strongest component of every bin (BeamformerEig's default).
        dict(plane256, name='eig_256mic', kind='eig', bin_lo=150, bins=16),
        # Functional beamforming: every eigenvalue and eigenvector of many bins and the map of all components.
        dict(name='functional_112mic', kind='functional', mics=112, radius=0.5, nx=61, ny=61, nz=1, extent=1.2,
             z=-0.7, steer='true location', r_diag=False, block=256, bin_lo=8, bins=64, gamma=4.0),
        # Deconvolution of the 8 kHz third-octave band by CLEAN-SC with its defaults.
        dict(band64, name='cleansc_64mic', kind='cleansc', n_iter=0),
        # Deconvolution of the same band by DAMAS with its defaults: maps, point-spread functions, 100 sweeps.
        dict(band64, name='damas_64mic', kind='damas', n_iter=100),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_recording(rng, c, max_mics, max_values):
    c['mics'] = _log_int(rng, 8, max_mics)
    c['block'] = rng.choice(BLOCKS)
    c['samples'] = max(2 * c['block'], min(_log_int(rng, 20000, 512000), max_values // c['mics']))
    c['dtype'] = rng.choice(('float32', 'float64'))
    c['window'] = rng.choice(('Rectangular', 'Hanning', 'Hamming', 'Bartlett', 'Blackman'))
    c['overlap'] = rng.choice(('None', '50%', '75%'))


def _draw_geometry(rng, c, lo_mics, hi_mics, lo_grid, hi_grid):
    c['mics'] = _log_int(rng, lo_mics, hi_mics)
    g = _log_int(rng, lo_grid, hi_grid)
    if rng.random() < 0.3:
        c['nx'] = max(2, int(round(g ** (1 / 3) * rng.uniform(0.8, 1.3))))
        c['ny'] = max(2, int(round(g ** (1 / 3) * rng.uniform(0.8, 1.3))))
        c['nz'] = max(2, int(round(g / (c['nx'] * c['ny']))))
    else:
        c['nx'] = max(2, int(round(g ** 0.5 * rng.uniform(0.7, 1.4))))
        c['ny'] = max(2, int(round(g / c['nx'])))
        c['nz'] = 1
    c['radius'] = round(rng.uniform(0.2, 0.8), 3)
    c['extent'] = round(rng.uniform(0.4, 2.0), 3)
    c['z'] = round(rng.uniform(0.3, 1.5) * rng.choice((-1, 1)), 3)
    c['steer'] = rng.choice(STEER)
    c['r_diag'] = rng.random() < 0.7
    if rng.random() < 0.2:
        c['ref'] = round(rng.uniform(0.05, 0.3), 3)


def _draw_bins(rng, c, most):
    c.setdefault('block', rng.choice(BLOCKS[:6]))
    f = c['block'] // 2
    c['bins'] = min(_log_int(rng, 1, most), f // 2)
    c['bin_lo'] = rng.randint(max(1, f // 32), max(1, f // 32, f * 3 // 4 - c['bins']))


def draw(rng):
    """One more case of the ranges that the listed ones stand for, no more work than the largest of its kind."""
    while True:
        c = {'kind': rng.choice(('analysis', 'csm', 'csm', 'map', 'map', 'map_tc', 'eig', 'functional', 'cleansc',
                                 'damas'))}
        if c['kind'] == 'csm':
            c['precision'] = rng.choice(('complex128', 'complex64', 'tc_tf32', 'tc_bf16x3'))
            _draw_recording(rng, c, 256, 512000 * 256)
        elif c['kind'] == 'analysis':
            c['precision'] = rng.choice(('complex128', 'complex64'))
            _draw_geometry(rng, c, 16, 128, 400, 6000)
            m = c['mics']
            _draw_recording(rng, c, 128, 8 << 20)
            c['mics'] = m
            c['block'] = rng.choice(BLOCKS[:5])
            _draw_bins(rng, c, 16)
        elif c['kind'] == 'map':
            c['form'] = 'f64'
            _draw_geometry(rng, c, 8, 512, 400, 161000)
            _draw_bins(rng, c, 64)
        elif c['kind'] == 'map_tc':
            c['kind'] = 'map'
            c['form'] = rng.choice(('bf16x3', 'tf32', 'fp16'))
            _draw_geometry(rng, c, 24, 1024, 1600, 161000)
            _draw_bins(rng, c, 256)
        elif c['kind'] == 'eig':
            _draw_geometry(rng, c, 16, 256, 1600, 161000)
            _draw_bins(rng, c, 32)
        elif c['kind'] == 'functional':
            _draw_geometry(rng, c, 16, 128, 900, 6000)
            _draw_bins(rng, c, 64)
            c['r_diag'] = False
            c['gamma'] = rng.choice((1.0, 3.0, 4.0, 10.0))
        elif c['kind'] == 'cleansc':
            _draw_geometry(rng, c, 16, 112, 400, 4000)
            _draw_bins(rng, c, 8)
            c['n_iter'] = rng.choice((0, 20, 60))
        else:
            _draw_geometry(rng, c, 16, 112, 400, 2000)
            _draw_bins(rng, c, 8)
            c['n_iter'] = rng.choice((20, 50, 100))
        most = [work(q) for q in listed() if q['kind'] == c['kind'] and (q.get('form') == 'f64') == (c.get('form') == 'f64')]
        w = work(c)
        if (w['flops'] <= max(q['flops'] for q in most) and w['bytes'] <= max(q['bytes'] for q in most)) or \
                (c['kind'] == 'analysis' and w['flops'] <= 2e10):
            return c


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _frequencies(case):
    return np.arange(case['block'] // 2 + 1) * (FS / case['block'])


def _geometry(case, seed):
    mics = disk_mics(case['mics'], case['radius'], seed=seed % (1 << 31))
    ext, z = case['extent'], case['z']
    x, y = (np.linspace(-ext / 2, ext / 2, case[k]) for k in ('nx', 'ny'))
    zz = np.linspace(z, z * 1.6, case['nz']) if case['nz'] > 1 else np.array([z])
    grid = np.ascontiguousarray(np.stack([a.ravel() for a in np.meshgrid(x, y, zz, indexing='ij')]))
    return mics.pos.astype(np.float64), grid


def _norm(case):
    return case['mics'] / (case['mics'] - 1.0) if case['r_diag'] else 1.0


def _ref(case):
    return np.array([case['ref'], 0.0, 0.0]) if 'ref' in case else 0.0


def _sources(case, grid, seed):
    """Five point sources on the grid, 0 to -20 dB."""
    r = np.random.RandomState(seed % (1 << 31))
    loc = grid[:, r.randint(0, grid.shape[1], 5)]
    return loc, 10 ** (-np.linspace(0, 20, 5) / 20)


def _csm(case, mpos, grid, seed):
    """CSM (bins, M, M) of the sources in uncorrelated channel noise, an average over 2 M + 32 snapshots."""
    dev = 'cuda'
    gen = torch.Generator(device=dev).manual_seed(seed)
    loc, amp = _sources(case, grid, seed)
    m, k_snap = case['mics'], 2 * case['mics'] + 32
    f = _frequencies(case)[case['bin_lo']:case['bin_lo'] + case['bins']]
    r = torch.as_tensor(np.linalg.norm(mpos[:, :, None] - loc[:, None, :], axis=0), device=dev)       # (M, 5)
    out = torch.empty((case['bins'], m, m), dtype=torch.complex128, device=dev)
    for b0 in range(0, case['bins'], 64):
        k = torch.as_tensor(2 * np.pi * f[b0:b0 + 64] / C0, device=dev)
        n = k.numel()
        a = torch.polar((torch.as_tensor(amp, device=dev) / r).expand(n, m, 5).contiguous(), -(k[:, None, None] * r))
        q = torch.randn((n, 5, k_snap), dtype=torch.complex128, device=dev, generator=gen)
        x = a @ q + 0.2 * torch.randn((n, m, k_snap), dtype=torch.complex128, device=dev, generator=gen)
        c = (x @ x.mH) / k_snap
        out[b0:b0 + n] = 0.5 * (c + c.mH)
    return out


def _samples(case, seed):
    """Recording (samples, channels): delayed broadband sources and sensor noise, a few hundredths to about 1 Pa."""
    dev = 'cuda'
    gen = torch.Generator(device=dev).manual_seed(seed)
    s, m = case['samples'], case['mics']
    x = 0.1 * torch.randn((s, m), dtype=torch.float32, device=dev, generator=gen)
    delay = torch.randint(0, 120, (3, m), device=dev, generator=gen)
    for j in range(3):
        sig = (0.5 / (j + 1)) * torch.randn(s + 120, dtype=torch.float32, device=dev, generator=gen)
        for i in range(0, s, 65536):
            t = torch.arange(i, min(i + 65536, s), device=dev)
            x[i:i + 65536] += sig[t[:, None] + delay[j][None, :]]
    return x.to(getattr(torch, case['dtype']))


def prepare(case, seed):
    kind = case['kind']
    st = {'case': case}
    if kind in ('csm', 'analysis', 'synthetic'):
        st['samples'] = _samples(case, seed)
    if kind == 'csm':
        return st
    mpos, grid = _geometry(case, seed)
    if kind == 'synthetic':
        st['samples'] = st['samples'].cpu().numpy()
        st['mics'] = ac.MicGeom(pos_total=mpos)
        ext = case['extent']
        st['grid'] = ac.RectGrid(x_min=-ext / 2, x_max=ext / 2, y_min=-ext / 2, y_max=ext / 2, z=case['z'],
                                 increment=ext / (case['nx'] - 1))
        return st
    f = _frequencies(case)[case['bin_lo']:case['bin_lo'] + case['bins']]
    st['k'] = torch.as_tensor(2 * np.pi * f / C0, device='cuda')
    st['mpos'], st['gpos'] = torch.as_tensor(mpos, device='cuda'), torch.as_tensor(grid, device='cuda')
    if kind != 'analysis':
        st['csm'] = _csm(case, mpos, grid, seed)
    if kind == 'damas':
        rm = torch.linalg.vector_norm(st['gpos'][:, :, None] - st['mpos'][:, None, :], dim=0)
        st['rm'] = rm.contiguous()
        st['r0'] = torch.linalg.vector_norm(st['gpos'] - torch.as_tensor(_ref_point(case), device='cuda')[:, None], dim=0)
    return st


def _ref_point(case):
    return np.asarray(_ref(case)) * np.ones(3) if np.isscalar(_ref(case)) else _ref(case)


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def run(st):
    case = st['case']
    kind = case['kind']
    if kind == 'csm':
        return D.calc_csm(st['samples'], case['block'], case['window'], case['overlap'], case['precision'])
    if kind == 'synthetic':
        ts = ac.TimeSamples(data=st['samples'], sample_freq=FS)
        ps = ac.PowerSpectra(source=ts, block_size=case['block'], window=case['window'], overlap=case['overlap'],
                             precision=case['precision'])
        sv = ac.SteeringVector(grid=st['grid'], mics=st['mics'], steer_type=case['steer'])
        return ac.BeamformerBase(freq_data=ps, steer=sv, r_diag=case['r_diag']).synthetic(8000, 3)
    geo = (st['mpos'], st['gpos'])
    args = (case['steer'], case['r_diag'], _norm(case))
    if kind == 'analysis':
        csm = D.calc_csm(st['samples'], case['block'], case['window'], case['overlap'], case['precision'])
        sub = csm[case['bin_lo']:case['bin_lo'] + case['bins']]
        return {'csm': csm, 'map': D.map_f64(sub, st['k'], *geo, *args, ref=_ref(case))}
    csm = st['csm']
    if kind == 'map':
        if case['form'] == 'f64':
            return D.map_f64(csm, st['k'], *geo, *args, ref=_ref(case))
        return D.map_tc(csm, st['k'], *geo, *args, ref=_ref(case), precision=case['form'])
    if kind == 'eig':
        lam, vec = D.heevd_select_f64(csm, [case['mics'] - 1])
        return {'eigval': lam, 'map': D.map_eig_f64(lam, vec, st['k'], *geo, *args, ref=_ref(case))}
    if kind == 'functional':
        ev, vec, info = D.heevd_f64(csm)
        sn = torch.empty((case['bins'], st['gpos'].shape[1]), dtype=torch.float64, device=csm.device)
        lam = ev.pow(1.0 / case['gamma']).contiguous()
        out = D.map_eig_f64(lam, vec, st['k'], *geo, case['steer'], False, 1.0, ref=_ref(case), steer_norm=sn)
        return {'eigval': ev, 'info': info, 'map': out.div_(sn).pow_(case['gamma']).mul_(sn)}
    if kind == 'cleansc':
        return D.cleansc_f64(csm, st['k'], *args, n_iter=case['n_iter'], mpos=st['mpos'], gpos=st['gpos'],
                             ref=_ref(case))
    y = D.map_f64(csm, st['k'], *geo, *args, ref=_ref(case), clip_negative=True)
    g = st['gpos'].shape[1]
    psf = torch.empty((case['bins'], g, g), dtype=torch.float64, device=csm.device)
    src = torch.arange(g, device=csm.device)
    f = _frequencies(case)
    for j in range(case['bins']):
        D.psf_f64(st['r0'], st['rm'], 2 * np.pi * f[case['bin_lo'] + j] / C0, src, case['steer'], out=psf[j])
    return {'map': y, 'solution': D.damas_gauss_seidel(psf, y, case['n_iter'], 1.0)}


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def work(case):
    kind, m = case['kind'], case['mics']
    by = fl = 0.0
    if kind in ('csm', 'analysis', 'synthetic'):
        n, s = case['block'], case['samples']
        win = (s - n) // (n // OVERLAP[case['overlap']]) + 1
        f = n // 2 + 1
        by += s * m * (4 if case['dtype'] == 'float32' else 8) + (0 if kind == 'synthetic' else 16.0 * f * m * m)
        fl += 2.5 * n * math.log2(n) * m * win + 4.0 * m * m * win * f
        if kind == 'csm':
            return {'bytes': by, 'flops': fl}
    g, b = case['nx'] * case['ny'] * case['nz'], case['bins']
    by += 8.0 * (3 * g + 3 * m + (b + 1) * g)
    if kind not in ('analysis', 'synthetic'):
        by += 16.0 * b * m * m
    quad = (4.0 * m * m + 8.0 * m) * g * b                # the Hermitian half of h^H C h
    if kind in ('map', 'analysis', 'synthetic'):
        fl += quad
    elif kind == 'eig':
        fl += 16.0 / 3 * m ** 3 * b + 8.0 * m * g * b
    elif kind == 'functional':
        fl += 24.0 * m ** 3 * b + 8.0 * m * m * g * b
    elif kind == 'cleansc':
        fl += quad + (case['n_iter'] or 2 * m) * b * (8.0 * m * g + 16.0 * m * m)
    else:
        fl += quad + b * (8.0 * m * g * g + 2.0 * case['n_iter'] * g * g)
    return {'bytes': by, 'flops': fl}


# ------------------------------------------------------------------------------------------------
# the same results in 64 bits, in plain torch and numpy
# ------------------------------------------------------------------------------------------------
def _exact_csm(x, case):
    n, ov = case['block'], OVERLAP[case['overlap']]
    hop = n // ov
    s, m = x.shape
    k = (s - n) // hop + 1
    w = {'Rectangular': np.ones, 'Hanning': np.hanning, 'Hamming': np.hamming, 'Bartlett': np.bartlett,
         'Blackman': np.blackman}[case['window']](n)
    wd = torch.as_tensor(w, device=x.device)
    out = torch.zeros((n // 2 + 1, m, m), dtype=torch.complex128, device=x.device)
    step = max(1, (1 << 26) // (n * m))
    for w0 in range(0, k, step):
        w1 = min(k, w0 + step)
        seg = x[w0 * hop:(w1 - 1) * hop + n].to(torch.float64).unfold(0, n, hop)          # (w, M, N)
        q = torch.fft.rfft(seg * wd, dim=2).permute(2, 1, 0)                              # (F, M, w)
        out += q @ q.mH
    return out * (2.0 / n / float(np.dot(w, w)) / (ov * s / n - ov + 1))


def _steering(case, kk, gpos, mpos, exact_phase):
    """Steering values e^{-i k r} (G, M), distances (G, M) and reference distances (G,); the phase rounded to single
    precision as the method defines it, except for the tensor-core forms, which do not round it."""
    r = torch.linalg.vector_norm(gpos[:, :, None] - mpos[:, None, :], dim=0)
    r0 = torch.linalg.vector_norm(gpos - torch.as_tensor(_ref_point(case), device=gpos.device)[:, None], dim=0)
    p = kk * r
    if not exact_phase:
        p = p.float().double()
    return torch.complex(torch.cos(p), -torch.sin(p)), r, r0


def _weights(case, h, r, r0):
    """Weighted steering values and the divisor of the quadratic form for the steering type."""
    m = case['mics']
    if case['steer'] == 'classic':
        return h, torch.full_like(r0, float(m) ** 2), torch.full_like(r0, 1.0 / m)
    if case['steer'] == 'inverse':
        return h * r, (m * r0) ** 2, (r * r).sum(1) / (m * r0) ** 2
    s = (1.0 / (r * r)).sum(1)
    if case['steer'] == 'true level':
        return h / r, (r0 * s) ** 2, 1.0 / (r0 * r0 * s)
    return h / r, m * s, torch.full_like(r0, 1.0 / m)


def _exact_map(case, csm, ks, gpos, mpos, exact_phase=False, clip=None, eig=None, gamma=None):
    g = gpos.shape[1]
    out = torch.empty((len(ks), g), dtype=torch.float64, device=gpos.device)
    step = max(1, (1 << 25) // case['mics'])
    for g0 in range(0, g, step):
        gp = gpos[:, g0:g0 + step].contiguous()
        for j, kk in enumerate(ks):
            h, r, r0 = _steering(case, kk, gp, mpos, exact_phase)
            v, div, sn = _weights(case, h, r, r0)
            if eig is None:
                c = csm[j].clone()
                if case['r_diag']:
                    c.diagonal().zero_()
                q = ((v.conj() @ c) * v).sum(1).real
            else:
                t = v.conj() @ eig[1][j]
                q = (t.real ** 2 + t.imag ** 2) @ eig[0][j]
                if case['r_diag']:
                    w = (eig[1][j].real ** 2 + eig[1][j].imag ** 2) @ eig[0][j]
                    q = q - (v.real ** 2 + v.imag ** 2) @ w
            q = q / div * _norm(case)
            out[j, g0:g0 + step] = (q / sn) ** gamma * sn if gamma else q
    if case['r_diag'] if clip is None else clip:
        out.clamp_(min=0.0)
    return out


def _exact_damas(case, y, ks, gpos, mpos):
    """Gauss-Seidel sweeps on the host, all bins at once."""
    g, b = gpos.shape[1], len(ks)
    a = np.empty((b, g, g))
    for j, kk in enumerate(ks):
        r = torch.linalg.vector_norm(gpos[:, :, None] - mpos[:, None, :], dim=0)
        r0 = torch.linalg.vector_norm(gpos - torch.as_tensor(_ref_point(case), device=gpos.device)[:, None], dim=0)
        for s0 in range(0, g, 256):
            rs = r[s0:s0 + 256]
            p = (kk * (r[:, None, :] - rs[None, :, :])).float().double()                  # (G, s, M)
            e = torch.complex(torch.cos(p), -torch.sin(p)) / rs[None]
            m = case['mics']
            if case['steer'] == 'classic':
                q = e.sum(2).abs() ** 2 * (r0[s0:s0 + 256][None] / m) ** 2
            elif case['steer'] == 'inverse':
                q = (e * r[:, None, :]).sum(2).abs() ** 2 * (r0[s0:s0 + 256][None] / r0[:, None] / m) ** 2
            else:
                h2 = (1.0 / (r * r)).sum(1)[:, None]
                q = (e / r[:, None, :]).sum(2).abs() ** 2 * r0[s0:s0 + 256][None] ** 2
                q = q / (r0[:, None] * h2) ** 2 if case['steer'] == 'true level' else q / m / h2
            a[j, :, s0:s0 + 256] = q.cpu().numpy()
    yy = y.cpu().numpy()
    x = yy.copy()
    rows = np.ascontiguousarray(a.transpose(1, 0, 2))                                      # (G, b, G)
    diag = np.ascontiguousarray(np.einsum('bgg->gb', a))
    for _ in range(case['n_iter']):
        for i in range(g):
            s = np.einsum('bg,bg->b', rows[i], x) - diag[i] * x[:, i]
            x[:, i] = np.maximum(0.0, yy[:, i] - s)
    return torch.from_numpy(x)


def exact(case, seed):
    kind = case['kind']
    if kind == 'cleansc':
        return None     # a sequence of argmax decisions: not a formula of the inputs
    st = prepare(case, seed)
    if kind == 'csm':
        return _exact_csm(st['samples'], case)
    if kind == 'synthetic':
        x = torch.from_numpy(st['samples']).cuda()
        f = _frequencies(case)
        lo, hi = (int(np.searchsorted(f, 8000 * 2.0 ** (e / 6))) for e in (-1, 1))
        out = _exact_map(case, _exact_csm(x, case)[lo:hi], 2 * np.pi * f[lo:hi] / C0,
                         torch.as_tensor(st['grid'].pos, device='cuda'), torch.as_tensor(st['mics'].pos, device='cuda'))
        return out.sum(0).reshape(st['grid'].shape).cpu().numpy()
    ks = st['k'].tolist()
    geo = (st['gpos'], st['mpos'])
    if kind == 'analysis':
        csm = _exact_csm(st['samples'], case)
        return {'csm': csm, 'map': _exact_map(case, csm[case['bin_lo']:case['bin_lo'] + case['bins']], ks, *geo)}
    if kind == 'map':
        return _exact_map(case, st['csm'], ks, *geo, exact_phase=case['form'] != 'f64')
    if kind == 'eig':
        ev, vec = torch.linalg.eigh(st['csm'])
        ev, vec = ev[:, -1:].contiguous(), vec[:, :, -1:].contiguous()
        return {'eigval': ev, 'map': _exact_map(case, None, ks, *geo, eig=(ev, vec))}
    if kind == 'functional':
        ev, vec = torch.linalg.eigh(st['csm'])
        p = (ev ** (1.0 / case['gamma'])).contiguous()
        return {'eigval': ev, 'info': None, 'map': _exact_map(case, None, ks, *geo, eig=(p, vec), gamma=case['gamma'])}
    y = _exact_map(case, st['csm'], ks, *geo, clip=True)
    if case['n_iter'] * st['gpos'].shape[1] * case['bins'] > 1_000_000:
        return {'map': y, 'solution': None}
    return {'map': y, 'solution': _exact_damas(case, y, ks, *geo)}
