"""The work that users of this framework have it do, as cases that can be timed and checked.

A case is a dict of plain values.  ``listed()`` names twelve, ``draw(rng)`` gives one more of
the same ranges, ``prepare(case, seed)`` makes what a user's program holds before the call,
``run(state)`` is one pass through the public entry points, ``work(case)`` the bytes and
operations that a pass cannot do without, and ``exact(case, seed)`` the same results in
64-bit arithmetic from plain torch.

Kinds:
* ``surface``: one ``OceanSurface.t`` assignment, every requested field on the device.
* ``pulse``: a window of pulses of ``RawGenerator.pulse`` on given surface fields (the
  stage-wise use: fields from elsewhere, or a frozen sea), raw rows and NRCS sums out.
* ``accum``: ``chan_profile_numba`` on device arrays, on a surface or on flattened facets.
* ``scene``: a whole short ``RawGenerator`` acquisition, surface synthesis included, by
  ``run`` or replayed from its CUDA graph.
* ``batch``: several scenes of uneven size driven to their end by ``SceneBatch``.
"""
import math
import os
import tempfile

import numpy as np
import torch

from oceansar_b200 import swell_spec
from oceansar_b200.radarsim.batch import SceneBatch
from oceansar_b200.radarsim.range_profile import calc_sinc_vec, chan_profile_numba
from oceansar_b200.radarsim.sar_raw_nompi import RawGenerator
from oceansar_b200.surfaces import OceanSurface

C_LIGHT = 2.99792458e8
FIELDS = ('Dx', 'Dy', 'Dz', 'Diffx', 'Diffy', 'Diffxx', 'Diffyy', 'Diffxy')
GROUPS = {'D': ('Dx', 'Dy', 'Dz'), 'Diff': ('Diffx', 'Diffy'), 'Diff2': ('Diffxx', 'Diffyy', 'Diffxy'),
          'V': ('Vx', 'Vy', 'Vz'), 'A': ('Ax', 'Ay', 'Az')}

CFG = """[sar]
f0=5.405e9
inc_angle={inc}
pol={pol}
squint=0
prf={prf}
rg_bw=50e6
over_fs=1.1
alt=514e3
v_ground=7600.
heading=0.
ant_L_tx={ant_l}
ant_L_rx={ant_l}
num_ch={num_ch}
b_ati={b_ati}
b_xti={b_xti}
[ocean]
Lx={Lx}
Ly={Ly}
dx={d}
dy={d}
opt_res=True
fft_max_prime={prime}
dt=0.05
depth=1e5
wind_dir={wind_dir}
wind_U={wind}
wind_fetch=500e3
swell_dir_enable={swell}
sigf=0.007
freq_r=0.07901333615718642
dir_swell_dir=120
sigs=8
Hs=0.8
swell_enable=False
swell_wl=60
swell_dir=20
swell_ampl=0.3
spec_model=elfouhaily
spread_model=cos2s
cutoff_wl=auto
current_mag=0
current_dir=0.
choppy_enable=False
frozen_ocean=False
[srg]
use_hmtf=False
nesz=-300.
wh_tol=2.73
scat_spec_enable={spec}
scat_spec_mode=kodis
scat_bragg_enable=True
scat_bragg_model=romeiser97
scat_bragg_spec=elfouhaily
scat_bragg_spread={spread}
scat_bragg_d=0.125
use_lut=False
"""


def _surface(name, nx, ny, groups, d=1.0, wind=7.0, prime=2, choppy=False, swell=False, dir_swell=False):
    return dict(name=name, kind='surface', nx=nx, ny=ny, groups=groups, d=d, wind=wind, prime=prime,
                choppy=choppy, swell=swell, dir_swell=dir_swell)


def _sar(name, kind, nx, ny, pulses, precision, ch=1, xti=False, pol='vv', wind=7.0, inc=35.0, d=1.0, prime=2,
         prf=1500.0, ant_l=2.742, swell=False, spec=True, spread='cos2s'):
    return dict(name=name, kind=kind, nx=nx, ny=ny, pulses=pulses, precision=precision, ch=ch, xti=xti, pol=pol,
                wind=wind, inc=inc, d=d, prime=prime, prf=prf, ant_l=ant_l, swell=swell, spec=spec, spread=spread)


def listed():
    return [
        # the 4096^2 stress scene's sea state at 0.5 m with directional swell: the largest
        # surface, the standard eight fields
        _surface('surface_4096', 4096, 4096, 'D Diff Diff2', d=0.5, wind=15.0, dir_swell=True),
        # the two-channel benchmark's surface at one pulse
        _surface('surface_2048', 2048, 2048, 'D Diff Diff2'),
        # a steep sea for Doppler studies on a ragged grid: choppy waves, a swell train,
        # velocities, mixed-radix transforms
        _surface('surface_ragged', 1200, 900, 'D Diff Diff2 V', wind=12.0, prime=5, choppy=True, swell=True),
        # the smallest calls: a 256^2 scene pulse by pulse, where launches count
        _sar('pulse_256', 'pulse', 256, 256, 8, 'mixed', wind=10.0, inc=12.0, prf=1000.0, ant_l=35.7),
        # the two-channel along-track benchmark scene, mixed precision
        _sar('pulse_2048_2ch', 'pulse', 2048, 2048, 16, 'mixed', ch=2),
        # along- and cross-track interferometer: four channels with an XTI baseline
        _sar('pulse_1024_xti', 'pulse', 1024, 1024, 16, 'mixed', ch=4, xti=True, wind=15.0, prf=2000.0,
             ant_l=1.7633),
        # the float64 drop-in (sar_raw's default), two channels, both polarisations, near-nadir
        # incidence and a rough sea: many specular facets
        _sar('pulse_f64_1024_dp', 'pulse', 1024, 1024, 8, 'f64', ch=2, pol='DP', wind=15.0, inc=12.0),
        # chan_profile_numba on a whole surface
        dict(name='accum_2d', kind='accum', rows=4096, cols=4096, d=0.5, inc=35.0, bins=2048, taps=8, ovs=20),
        # chan_profile_numba as the reference calls it: one flattened list of facets
        dict(name='accum_flat', kind='accum', rows=0, cols=2999999, d=0.5, inc=35.0, bins=4096, taps=8, ovs=20),
        # the one-channel 512^2 acquisition by the generator's run() in sar_raw's default
        # precision, as sar_raw does it
        _sar('scene_512_run', 'scene', 512, 512, 48, 'f64', wind=10.0, prf=1000.0, ant_l=35.7),
        # the benchmark scene's acquisition replayed from its CUDA graph
        dict(_sar('scene_2048_graph', 'scene', 2048, 2048, 16, 'mixed', ch=2), graph=True),
        # the batched workload: six scenes of 256^2 to 1024^2 side by side
        dict(name='batch_6', kind='batch', scenes=6, pulses=24, most=1024, pick=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['surface', 'surface', 'pulse', 'pulse', 'pulse', 'accum', 'accum', 'scene', 'batch'])
    prime = rng.choice([2, 2, 5])
    if kind == 'surface':
        c = _surface('', _log(rng, 128, 3000), _log(rng, 128, 2048),
                     rng.choice(['D Diff Diff2', 'D Diff Diff2', 'D Diff', 'D Diff Diff2 V', 'D V A']),
                     d=rng.choice([0.5, 1.0]), wind=round(rng.uniform(4., 15.), 2), prime=prime,
                     choppy=rng.random() < 0.2, swell=rng.random() < 0.3)
    elif kind == 'pulse':
        prec, pol = rng.choice(['mixed', 'mixed', 'f64']), rng.choice(['vv', 'vv', 'hh', 'DP'])
        most = 2048 if (prec, pol) in (('mixed', 'vv'), ('mixed', 'hh')) else 1024
        c = _sar('', 'pulse', _log(rng, 200, most), _log(rng, 200, most), rng.randint(4, 16), prec,
                 ch=rng.randint(1, 4), xti=rng.random() < 0.3, pol=pol, wind=round(rng.uniform(3., 15.), 2),
                 inc=round(rng.uniform(12., 45.), 2), prime=prime, prf=rng.choice([1000.0, 1500.0, 2000.0]),
                 spec=rng.random() < 0.8, spread=rng.choice(['cos2s', 'elfouhaily']))
    elif kind == 'accum':
        flat = rng.random() < 0.5
        c = dict(kind='accum', rows=0 if flat else _log(rng, 50, 4096),
                 cols=_log(rng, 10000, 4000000) if flat else _log(rng, 50, 4096), d=rng.choice([0.5, 1.0]),
                 inc=round(rng.uniform(20., 45.), 2), bins=rng.choice([512, 1000, 2048, 4096]),
                 taps=rng.choice([8, 8, 8, 10, 6]), ovs=rng.choice([20, 20, 10]))
    elif kind == 'scene':
        prec = rng.choice(['mixed', 'f64'])
        most = 1024 if prec == 'mixed' else 512
        c = _sar('', 'scene', _log(rng, 128, most), _log(rng, 128, most), rng.randint(12, 32), prec,
                 ch=rng.randint(1, 3), wind=round(rng.uniform(3., 15.), 2), inc=round(rng.uniform(20., 45.), 2),
                 prime=prime, prf=1000.0)
        c['graph'] = rng.random() < 0.5
    else:
        c = dict(kind='batch', scenes=rng.randint(3, 8), pulses=rng.randint(12, 24), most=rng.choice([512, 1024]),
                 pick=rng.randint(0, 10 ** 6))
    c.pop('name', None)
    return c


# ---- what a user's program holds before the call ------------------------------------------
def _device():
    return torch.device('cuda' if torch.cuda.is_available() else 'cpu')


def _make_surface(c, seed, device):
    np.random.seed(seed)
    s = OceanSurface()
    s.init(c['nx'] * c['d'], c['ny'] * c['d'], c['d'], c['d'], 'auto', 'elfouhaily', 'cos2s', np.deg2rad(45.), 500e3,
           c['wind'], 0.5 if c['choppy'] else 0., np.deg2rad(60.), dir_swell_dir=120,
           freq_r=0.07901333615718642, sigf=0.007, sigs=8, Hs=0.8, swell_dir_enable=c['dir_swell'],
           swell_enable=c['swell'], swell_ampl=0.3, swell_dir=np.deg2rad(20.), swell_wl=60.,
           compute=c['groups'].split(), fft_max_prime=c['prime'], choppy_enable=c['choppy'], depth=1e5,
           dir_swell_spec=swell_spec.ardhuin_swell_spec, device=device)
    return s


def _generator(c, seed, device):
    """The scene's RawGenerator: the .cfg file's set-up, numpy's generator seeded."""
    fd, path = tempfile.mkstemp(suffix='.cfg')
    n = c['ch']
    ati = '[' + ', '.join('%.1f' % (5.0 * (k % 3)) for k in range(n)) + ']' if n > 1 else '0.0'
    xti = '[' + ', '.join('%.1f' % (2.0 if k == n - 1 else 0.0) for k in range(n)) + ']' if n > 1 and c['xti'] else '0'
    try:
        with os.fdopen(fd, 'w') as f:
            f.write(CFG.format(Lx=c['nx'] * c['d'], Ly=c['ny'] * c['d'], b_ati=ati, b_xti=xti, num_ch=n, wind_dir=45.0,
                               **{k: c[k] for k in ('inc', 'pol', 'prf', 'ant_l', 'd', 'prime', 'wind', 'swell', 'spec',
                                                    'spread')}))
        return RawGenerator(path, precision=c['precision'], overrides=dict(az_steps=c['pulses']), seed=seed,
                            device=device)
    finally:
        os.unlink(path)


def _batch_scenes(c, seed, device):
    """The batch's scenes: grids, channels, incidence and lengths as the batched workload
    draws them, from the case; surfaces and scatterers from the seed."""
    r = np.random.default_rng(c['pick'])
    gens = []
    for k in range(c['scenes']):
        n = int(r.choice([g for g in (256, 512, 1024) if g <= c['most']]))
        sc = _sar('', 'scene', n, n, c['pulses'] + 4 * (k % 3), 'mixed', ch=int(r.integers(1, 4)),
                  wind=float(r.uniform(3., 20.)), inc=float(r.uniform(20., 45.)), prf=1000.0)
        gens.append(_generator(sc, (seed * 16 + k) % 2 ** 32, device))
    return gens


def _facets(c, seed):
    """Slant ranges and scene values of a sea surface's facets: ground-range columns with
    the waves' range offsets (metres) on top, complex Gaussian scattering coefficients."""
    g = torch.Generator(device=_device()).manual_seed(seed)
    mk = lambda *s: torch.randn(*s, generator=g, device=_device(), dtype=torch.float64)  # noqa: E731
    rows, cols = max(1, c['rows']), c['cols']
    width = cols if c['rows'] else max(64, int(math.sqrt(cols)))
    x = torch.arange(cols, device=_device(), dtype=torch.float64) % width
    srg = (x * c['d'] * math.sin(math.radians(c['inc'])))[None, :] + 0.4 * mk(rows, cols)
    if c['rows']:
        az = (torch.arange(rows, device=_device(), dtype=torch.float64) - rows / 2) * c['d'] + 3000.0
        srg = srg + (az * az / (2 * 6.1e5) - 3000.0 ** 2 / (2 * 6.1e5))[:, None]
    scene = torch.complex(mk(rows, cols), mk(rows, cols))
    return (srg, scene) if c['rows'] else (srg[0].contiguous(), scene[0].contiguous())


def prepare(case, seed):
    kind = case['kind']
    if kind == 'surface':
        s = _make_surface(case, seed, True)
        return dict(kind=kind, surface=s, t=0.37 + 0.01 * (seed % 7),
                    names=[f for g in ('D', 'Diff', 'Diff2', 'V', 'A') if g in case['groups'].split()
                           for f in GROUPS[g]])
    if kind == 'pulse':
        gen = _generator(case, seed, True)
        for n, f in zip(FIELDS, _linear_fields(gen.surface, 0.0, FIELDS if case['spec'] else FIELDS[:5])):
            gen.surface.field(n).copy_(f)
        return dict(kind=kind, gen=gen, pulses=case['pulses'])
    if kind == 'accum':
        srg, scene = _facets(case, seed)
        out = torch.zeros(case['bins'], dtype=torch.complex128, device=_device())
        return dict(kind=kind, srg=srg, scene=scene, out=out, binsize=C_LIGHT / (2 * 50e6) / 1.1, min_sr=-2.73,
                    sinc=calc_sinc_vec(case['taps'], case['ovs'], Fs=1.1), taps=case['taps'], ovs=case['ovs'])
    if kind == 'scene':
        gen = _generator(case, seed, True)
        if case.get('graph'):
            gen.capture()
        return dict(kind=kind, gen=gen, graph=bool(case.get('graph')))
    gens = _batch_scenes(case, seed, False)
    return dict(kind=kind, gens=gens, batch=SceneBatch(max_slots=len(gens), precision='mixed'))


def run(state):
    kind = state['kind']
    if kind == 'surface':
        s = state['surface']
        s.t = state['t']
        return [s.field(n) for n in state['names']]
    if kind == 'pulse':
        gen = state['gen']
        gen.reset()
        for a in range(state['pulses']):
            gen.pulse(a, update_surface=False)
        gen.flush()
        return [gen.raw_d, gen.nrcs_spec_d, gen.nrcs_bragg_d]
    if kind == 'accum':
        state['out'].zero_()
        chan_profile_numba(state['srg'], state['scene'], state['binsize'], state['min_sr'], state['sinc'],
                           state['taps'], state['ovs'], state['out'])
        return state['out']
    if kind == 'scene':
        gen = state['gen']
        if state['graph']:
            gen.replay()
        else:
            gen.reset()
            gen.run()
        return [gen.raw_d, gen.nrcs_spec_d, gen.nrcs_bragg_d]
    for gen in state['gens']:
        state['batch'].add(gen, tile_rows=32)
    state['batch'].run(pulse_block=8)
    return [[gen.raw_d, gen.nrcs_spec_d, gen.nrcs_bragg_d] for gen in state['gens']]


# ---- what a pass cannot do without --------------------------------------------------------
def _grid(c):
    s = _size(int(c['nx'] * c['d'] / c['d']), c['prime']), _size(int(c['ny'] * c['d'] / c['d']), c['prime'])
    return s[0] * s[1]


def _size(n, prime):
    def largest(v):
        p, best = 2, 1
        while v > 1:
            while v % p == 0:
                best, v = p, v // p
            p += 1
        return best
    if prime == 2:
        return 1 << (n - 1).bit_length()
    while largest(n) > prime:
        n += 1
    return n


def _fft_flops(facets, nfields):
    return 5.0 * facets * math.log2(facets) * nfields / 2


def _pulse_work(c, facets, synth):
    """One pulse: the fields (or, with the synthesis, the spectrum), the two scatterer start
    indices and sqrt(RCS) of every facet read, the raw rows written."""
    nf = 8 if c['spec'] else 5
    npol = 2 if c['pol'] == 'DP' else 1
    nout = npol * c['ch']
    real = 8 if c['precision'] == 'f64' else 4
    by = facets * ((12 if synth else 4 * nf) + 8 + 2 * npol * real) + nout * 1024 * 2 * real
    fl = facets * (60 + (50 if c['spec'] else 0) + 30 * npol + nout * (14 + 4 * 8))
    return by, fl + (_fft_flops(facets, nf) if synth else 0)


def work(case):
    kind = case['kind']
    if kind == 'surface':
        n = _grid(case)
        nf = sum(len(GROUPS[g]) for g in case['groups'].split())
        return {'bytes': float(n * (12 + 4 * nf)), 'flops': _fft_flops(n, nf)}
    if kind == 'accum':
        n = max(1, case['rows']) * case['cols']
        return {'bytes': float(24 * n + 32 * case['bins']), 'flops': float(n * (8 + 4 * case['taps']))}
    if kind == 'batch':
        r = np.random.default_rng(case['pick'])
        by = fl = 0.0
        for k in range(case['scenes']):
            n = int(r.choice([g for g in (256, 512, 1024) if g <= case['most']]))
            sc = dict(spec=True, pol='vv', ch=int(r.integers(1, 4)), precision='mixed')
            r.uniform(), r.uniform()            # wind and incidence, which change no work
            b, f = _pulse_work(sc, n * n, True)
            by, fl = by + b * (case['pulses'] + 4 * (k % 3)), fl + f * (case['pulses'] + 4 * (k % 3))
        return {'bytes': by, 'flops': fl}
    b, f = _pulse_work(case, _grid(case), kind == 'scene')
    return {'bytes': float(b * case['pulses']), 'flops': float(f * case['pulses'])}


# ---- the same results in 64-bit arithmetic ------------------------------------------------
def _t64(a):
    a = np.asarray(a)
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.complex128 if a.dtype.kind == 'c' else np.float64)).to(
        _device())


def _multiplier(name, kx, ky, kinv, om):
    return {'Dx': 1j * kx * kinv, 'Dy': 1j * ky * kinv, 'Dz': 1.0, 'Diffx': 1j * kx, 'Diffy': 1j * ky,
            'Diffxx': -kx * kx, 'Diffyy': -ky * ky, 'Diffxy': -kx * ky, 'Vx': kx * kinv * om, 'Vy': ky * kinv * om,
            'Vz': -1j * om, 'Ax': -1j * kx * kinv * om * om, 'Ay': -1j * ky * kinv * om * om, 'Az': -om * om,
            'xx': -kx * kx * kinv, 'yy': -ky * ky * kinv, 'xxx': -1j * kx ** 3 * kinv, 'yyy': -1j * ky ** 3 * kinv,
            'xxy': -1j * kx * kx * ky * kinv}[name]


def _linear_fields(s, t, names):
    """Re(ifft2(M c exp(-i omega t))) of every named field, float64."""
    om = _t64(s.omega)
    # the phase omega t is a float32 product by definition of the surface
    ph = (torch.from_numpy(np.asarray(s.omega, np.float32)).to(_device()) * float(np.float32(t))).double()
    c = _t64(s.wave_coefs) * torch.polar(torch.ones_like(ph), -ph)
    kx, ky = _t64(s.kx_s)[None, :], _t64(s.ky_s)[:, None]
    k = torch.sqrt(kx * kx + ky * ky)
    kinv = torch.where(k > float(s.kmin_half), 1.0 / k, torch.zeros_like(k))
    for n in names:
        yield torch.fft.ifft2(_multiplier(n, kx, ky, kinv, om) * c).real


def _exact_surface(case, seed):
    s = _make_surface(case, seed, False)
    t = float(np.float32(0.37 + 0.01 * (seed % 7)))
    names = [f for g in ('D', 'Diff', 'Diff2', 'V', 'A') if g in case['groups'].split() for f in GROUPS[g]]
    out = dict(zip(names, _linear_fields(s, t, names)))
    if case['choppy'] and 'Diffx' in out:
        xx, yy, xxx, yyy, xxy = _linear_fields(s, t, ('xx', 'yy', 'xxx', 'yyy', 'xxy'))
        px, py, ax, ay = 1 + xx, 1 + yy, out['Diffx'], out['Diffy']
        out['Diffx'], out['Diffy'] = ax / px, ay / py
        if 'Diffxx' in out:
            out['Diffxx'] = (px * out['Diffxx'] - xxx * ax) / px ** 3
            out['Diffyy'] = (py * out['Diffyy'] - yyy * ay) / py ** 3
            out['Diffxy'] = (px * out['Diffxy'] - xxy * ax) / (px ** 2 * py)
    if case['swell']:
        kx, ky, k, om = (complex(getattr(s, n)) for n in ('swell_kx', 'swell_ky', 'swell_k', 'swell_omega'))
        sw = _t64(s.swell_exp) * complex(np.exp(-1j * om.real * t))
        for n in names:
            m = {'Dx': 1j * kx / k, 'Dy': 1j * ky / k, 'Dz': 1., 'Diffx': 1j * kx, 'Diffy': 1j * ky, 'Diffxx': -kx ** 2,
                 'Diffyy': -ky ** 2, 'Diffxy': -kx * ky, 'Vx': kx / k * om, 'Vy': ky / k * om, 'Vz': -1j * om,
                 'Ax': -1j * kx / k * om ** 2, 'Ay': -1j * ky / k * om ** 2, 'Az': -om ** 2}[n]
            out[n] = out[n] + (m * sw).real
    for n, v in (('Dx', s.current[0] * t), ('Dy', s.current[1] * t), ('Vx', s.current[0]), ('Vy', s.current[1])):
        if n in out:
            out[n] = out[n] + float(v)
    return [out[n] for n in names]


def _accumulate(srg, vals, binsize, min_sr, sinc, taps, ovs, nbins):
    """Range profiles of facets: vals [outputs, ...] into complex128 [outputs, nbins]."""
    bf = (srg - min_sr) / binsize
    fl = torch.floor(bf)
    lut = torch.round(ovs * (1 - (bf - fl))).long()
    first = fl.long() - taps // 2
    out = torch.zeros((len(vals), nbins + 1, 2), dtype=torch.float64, device=srg.device)
    for j in range(taps):
        b = first + j
        b = torch.where((b >= 0) & (b < nbins), b, torch.full_like(b, nbins)).reshape(-1)
        w = sinc[lut + j * ovs]
        for o, v in enumerate(vals):
            out[o].index_add_(0, b, torch.view_as_real(w * v).reshape(-1, 2))
    return torch.view_as_complex(out[:, :nbins].contiguous())


def _sea_water():
    return 73 + 18j


def _bragg_rcs(g, azp, diffx, diffy):
    """Composite Bragg cross sections of both lines: {'hh': [2], 'vv': [2]} of [ny, nx]."""
    m = g.rcs_bragg
    k0, eps = float(m.k0), _sea_water()
    inc = _t64(g.inc)
    sa, ca = torch.sin(azp), torch.cos(azp)
    sp = torch.atan(ca * diffx + sa * diffy)
    st = torch.atan(-sa * diffx + ca * diffy)
    ip = inc - sp
    sin_t2 = 1 - torch.cos(st) ** 2
    cos_th = torch.cos(ip) * torch.cos(st)
    sin_th2 = 1 - cos_th ** 2
    b_hh = eps / (cos_th + np.sqrt(eps)) ** 2
    b_vv = eps ** 2 * (1 + sin_th2) / (eps * cos_th + np.sqrt(eps)) ** 2
    w = torch.cos(ip) / (torch.cos(inc) * torch.cos(sp))
    a, b = sin_t2 / sin_th2, torch.sin(ip) ** 2 * torch.cos(st) ** 2 / sin_th2
    f0 = 8 * math.pi * (k0 * cos_th) ** 4
    t_vv, t_hh = w * f0 * (b * b_vv + a * b_hh).abs() ** 2, w * f0 * (b * b_hh + a * b_vv).abs() ** 2
    kb = 2 * k0 * torch.sqrt(torch.sin(ip) ** 2 + torch.cos(ip) ** 2 * sin_t2)
    kb = torch.where(kb > 2 * k0, torch.zeros_like(kb), kb)
    phi = azp + torch.atan(torch.cos(ip) * torch.sin(-st) / torch.sin(ip))
    tk, ts = _t64(m.interp_k), _t64(m.interp_S)
    i = torch.searchsorted(tk, kb).clamp(1, len(tk) - 1)
    s = (ts[i] - ts[i - 1]) / (tk[i] - tk[i - 1]) * (kb - tk[i - 1]) + ts[i - 1]
    s = torch.where((kb >= tk[0]) & (kb <= tk[-1]), s, torch.ones_like(s))
    lines = []
    for turn in (0.0, math.pi):
        th = phi + turn - float(m.wind_dir)
        th = torch.atan2(torch.sin(th), torch.cos(th))
        if m.sw_dir_func == 'cos2s':
            spread = torch.cos(th) ** 2 / math.pi
        else:
            ck_p, ck_m, a0, ap, am = (float(v) for v in m.spread_consts)
            ck = torch.sqrt(9.80665 / kb + 0.072 / 1000. * kb)
            d = torch.tanh(a0 + ap * (ck / ck_p) ** 2.5 + am * (ck_m / ck) ** 2.5)
            spread = (1 + d * torch.cos(2 * th)) / math.pi
        lines.append(s / kb * torch.where(th.abs() <= math.pi / 2, spread, torch.zeros_like(spread)))
    bad = 4 * torch.sin(ip) ** 2 < float(m.d) ** 2
    area = float(m.dx) * float(m.dy)
    zero = torch.zeros_like(t_vv)
    vv = [torch.where(bad, zero, t_vv * x * area) for x in lines]
    hh = [torch.where(bad, zero, t_hh * x * area) for x in lines]
    if g.pol == 'DP':                       # the model leaves line 0 of hh unmasked here
        hh[0] = t_hh * lines[0] * area
    return {'hh': hh, 'vv': vv}


def _kodis(g, srs, azp, f):
    """Stationary-phase specular field times sqrt(4 pi); the curvature determinant and the
    slope factor are float32 quantities by definition."""
    s = g.surface
    dx, dy, dxx, dyy, dxy = (f[n] for n in ('Diffx', 'Diffy', 'Diffxx', 'Diffyy', 'Diffxy'))
    f32 = lambda n: f[n].float()  # noqa: E731
    J = f32('Diffxx') * f32('Diffyy') - f32('Diffxy') * f32('Diffxy')
    fac = f32('Diffx') * f32('Diffx') + f32('Diffy') * f32('Diffy') + 1.0
    inc = _t64(g.inc)
    ty, tx = dy - torch.tan(inc) * torch.sin(azp), dx - torch.tan(inc) * torch.cos(azp)
    inv = (1.0 / J.abs()).double()
    px, py = inv * (dxy * ty - dyy * tx), inv * (dxy * tx - dxx * ty)
    inside = (px.abs() < float(s.dx) / 2) & (py.abs() < float(s.dy) / 2) & (J != 0)
    pz = px * dx + py * dy
    r = srs + (torch.sin(inc) * torch.cos(azp) * px + torch.sin(inc) * torch.sin(azp) * py - torch.cos(inc) * pz)
    eps = torch.where(J > 0, torch.sign(dxx).to(torch.complex128), torch.full_like(dxx, 1.0).to(torch.complex128) * 1j)
    R = (_sea_water() - np.sqrt(_sea_water())) / (_sea_water() + np.sqrt(_sea_water()))
    ph = (-2 * g.k0) * r
    e = R / 2 * eps * fac.double() * torch.polar(torch.ones_like(ph), ph) / torch.sqrt(J.abs()).double()
    e = e * math.sqrt(4 * math.pi)
    return torch.where(inside, e, torch.zeros_like(e))


def _exact_raw(g, case, fields):
    """Raw rows [pol * ch, pulses, bins] and NRCS sums; fields(t) -> {name: float64}."""
    s, n = g.surface, case['pulses']
    sr, inc = _t64(g.sr), _t64(g.inc)
    sin_i, cos_i = _t64(g.sin_inc), _t64(g.cos_inc)
    sinc = _t64(g.chan_sinc_vec)
    pols = ['hh', 'vv'] if g.pol == 'DP' else [g.pol]
    raw = torch.zeros((len(pols) * g.num_ch, n, g.rg_samp), dtype=torch.complex128, device=_device())
    spec = torch.zeros(n, dtype=torch.float64, device=_device())
    bragg = torch.zeros((len(pols), n), dtype=torch.float64, device=_device())
    series = [(_t64(r.s), torch.from_numpy(np.asarray(r.ind0, np.int64)).to(_device()), int(r.N), r.Fs)
              for r in (g.rndscat_m, g.rndscat_p)]
    last, rcs = -1.0, None
    for a in range(n):
        t = a * g.t_step
        az = _t64(s.y)[:, None] - (t - g.t_span / 2.) * g.v_ground
        sin_az, azp = az / g.sr0, torch.asin(az / g.gr0)
        f = fields(t)
        srs = sr - cos_i * f['Dz']
        srs = srs + (az * 0.5) * sin_az
        srs = srs + f['Dx'] * sin_i
        srs = srs + f['Dy'] * sin_az
        scene = [torch.zeros_like(srs, dtype=torch.complex128) for _ in pols]
        if g.scat_spec_enable:
            e = _kodis(g, srs, azp, f)
            spec[a] = (e.abs() ** 2).sum()
            scene = [x + e for x in scene]
        if t - last > g.ocean_dt:
            rcs, last = _bragg_rcs(g, azp, f['Diffx'], f['Diffy']), t
            for p, pol in enumerate(pols):
                bragg[p, a] = rcs[pol][0].sum() + rcs[pol][1].sum()
        cap = 2 * g.k0 * g.t_step * _t64(g.c_b) * (a + 1)
        for k, (sign, (ser, ind0, N, fs)) in enumerate(zip((-1.0, 1.0), series)):
            ph = -2 * g.k0 * srs + sign * cap
            w = torch.polar(torch.ones_like(ph), ph) * ser[(ind0 + int(t * fs)) % N]
            for p, pol in enumerate(pols):
                scene[p] = scene[p] + torch.sqrt(rcs[pol][k]) * w
        pat = torch.sinc(g.ant_l_tx * g.f0 / C_LIGHT * sin_az) * torch.sinc(g.ant_l_rx * g.f0 / C_LIGHT * sin_az)
        vals = []
        for x in scene:
            for c in range(g.num_ch):
                ph = -g.k0 * float(g.b_ati[c]) * sin_az
                if g.b_xti[c] != 0:
                    ph = ph - g.k0 * float(g.b_xti[c]) * (inc - g.inc_angle + (f['Dz'] * sin_i + f['Dx'] * sin_i) / g.sr0)
                vals.append(x * pat * torch.polar(torch.ones_like(ph), ph))
        raw[:, a] = _accumulate(srs, vals, float(g.sr_res / g.over_fs), float(g.min_sr), sinc, 8, 20, g.rg_samp)
    return [raw, spec, bragg]


def _exact_scene(g, case):
    names = FIELDS if case['spec'] else FIELDS[:5]
    return _exact_raw(g, case, lambda t: dict(zip(names, _linear_fields(g.surface, t, names))))


def exact(case, seed):
    kind = case['kind']
    if kind == 'surface':
        return _exact_surface(case, seed)
    if kind == 'accum':
        srg, scene = _facets(case, seed)
        sinc = torch.from_numpy(calc_sinc_vec(case['taps'], case['ovs'], Fs=1.1)).double().to(_device())
        return _accumulate(srg, [scene], C_LIGHT / (2 * 50e6) / 1.1, -2.73, sinc, case['taps'], case['ovs'],
                           case['bins'])[0]
    if kind == 'pulse':
        g = _generator(case, seed, False)
        names = FIELDS if case['spec'] else FIELDS[:5]
        # the fields that the pulses were given: float32
        f = {n: v.float().double() for n, v in zip(names, _linear_fields(g.surface, 0.0, names))}
        return _exact_raw(g, case, lambda t: f)
    if kind == 'scene':
        return _exact_scene(_generator(case, seed, False), case)
    return [_exact_scene(g, dict(spec=True, pulses=int(g.az_steps))) for g in _batch_scenes(case, seed, False)]
