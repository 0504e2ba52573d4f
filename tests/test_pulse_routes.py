"""Which launches a mixed pulse takes, from the dispatch itself (no GPU needed: the descriptor's
pointers are never followed), at the limits of the fine grid's rule; and, on the GPU, the calls
beyond such a limit against the ones inside it."""
import ctypes

import numpy as np
import pytest

from oceansar_b200 import _capi
from oceansar_b200._structs import PulseDesc
from oceansar_b200.radarsim.sar_raw_nompi import PRECISIONS

GRID, WINDOWS = 1, 2                       # launches of an ordinary pulse: its kernel, or a row table before it


def route(precision='mixed', **kw):
    """Launches of an ordinary one-channel pulse on 128 x 64 facets of 1 m at 35 degrees."""
    zero = (ctypes.c_double * 1)(0.0)
    d = PulseDesc()
    kw = dict(dict(nx=128, ny=64, npol=1, pol=1, nch=1, az_steps=4, tind=3, inc_angle=np.deg2rad(35.), sr0=8e5, gr0=5e5,
                   k0=113.0, f0=5.4e9, binsize=2.725, t_step=1e-3, facet_dx=1.0, facet_dy=1.0, do_kodis=1, do_bragg=1,
                   n_m=5000, n_p=5000, spec_n=2, nbins=64), **kw)
    plane = 4 * kw['nx'] * kw['ny']
    for k, f in enumerate(('dx_d', 'dy_d', 'dz_d', 'diffx_d', 'diffy_d', 'diffxx_d', 'diffyy_d', 'diffxy_d')):
        setattr(d, f, 4096 + k * plane)
    for f, t in PulseDesc._fields_:
        if t is ctypes.c_void_p and f not in ('hmtf_d', 'lut_d', 'x_d') and not getattr(d, f):
            setattr(d, f, 1 << 40)
    for f, v in kw.items():
        setattr(d, f, v)
    d.b_ati = d.b_xti = ctypes.cast(zero, ctypes.POINTER(ctypes.c_double))
    return _capi.load().ocs_pulse_launches(ctypes.addressof(d), PRECISIONS[precision])


@pytest.mark.parametrize("n_m,n_p,launches", [
    (2 ** 29 - 1, 2 ** 29 - 1, GRID), (2 ** 29, 5000, WINDOWS), (5000, 2 ** 29, WINDOWS), (2 ** 30, 2 ** 30, WINDOWS)])
def test_series_that_32_bit_offsets_cannot_address(n_m, n_p, launches):
    assert route(n_m=n_m, n_p=n_p) == launches
    assert route(n_m=n_m, n_p=n_p, do_bragg=0) == GRID
    assert route('f64', n_m=n_m, n_p=n_p) == GRID          # 64-bit offsets


@pytest.mark.gpu
def test_long_series_on_the_gpu(tmp_path):
    """Scatterer series of more than 2^29 entries: the entries in use, moved past 2^29, give the
    same pulse (mixed against mixed, two routes: the bar of the mixed form)."""
    torch = pytest.importorskip("torch")
    from oceansar_b200.radarsim.sar_raw_nompi import RawGenerator
    from test_gpu_pulse_forms import make_cfg
    cfg = make_cfg(tmp_path, 128, 64, 1.0, 35.0, 'vv', 1, 0)
    raws = []
    for shift in (0, 2 ** 29):
        g = RawGenerator(cfg, precision='mixed', seed=3, overrides=dict(az_steps=60))
        if shift:
            keep = []
            for r, s32, ind0, n in (('rndscat_m', 's_m32_d', 'ind0_m_d', 'n_m'), ('rndscat_p', 's_p32_d', 'ind0_p_d', 'n_p')):
                s = getattr(g, r).device32().reshape(-1)
                idx = torch.from_numpy(np.asarray(getattr(g, r).ind0, np.int32)).cuda()
                length = shift + 2 * len(s)
                big = torch.zeros(length, dtype=torch.complex64, device='cuda')
                big[shift:shift + len(s)] = s
                big[shift + len(s):] = s
                idx = (idx + shift).contiguous()
                setattr(g.desc, s32, big.data_ptr())
                setattr(g.desc, ind0, idx.data_ptr())
                setattr(g.desc, n, length)
                keep += [big, idx]
        g.surface.set_t(0.1)
        for a in (0, 1, 59):
            g.pulse(a, update_surface=False)
        raws.append(g.raw()[:, :, [0, 1, 59]])
    assert np.abs(raws[0]).max() > 0
    assert np.linalg.norm(raws[1] - raws[0]) <= 1e-4 * np.linalg.norm(raws[0])


@pytest.mark.parametrize("d,inc,nx,ny,launches", [
    (1.0, 35., 2048, 2048, GRID), (0.5, 12., 2048, 2048, GRID), (0.139, 35., 2048, 2048, GRID),
    (0.139, -35., 2048, 2048, GRID), (0.138, 35., 2048, 2048, WINDOWS), (0.01, 35., 2048, 2048, WINDOWS),
    (0.01, 35., 128, 64, GRID), (0.009, 35., 128, 64, WINDOWS), (0.001, 35., 128, 64, WINDOWS),
    (0.05, 35., 1024, 512, GRID), (0.049, 35., 1024, 512, WINDOWS), (1.0, 4.6, 2048, 2048, GRID),
    (1.0, 4.5, 2048, 2048, WINDOWS), (1.0, 0., 128, 64, WINDOWS)])
def test_cells_of_many_facets(d, inc, nx, ny, launches):
    """Cells of at most 48 facets would need tiles of fewer rows than the pulse's own or 28."""
    assert route(facet_dx=d, inc_angle=np.deg2rad(inc), nx=nx, ny=ny) == launches


@pytest.mark.parametrize("d,inc,launches", [
    (1.0, 35., GRID), (0.0186, 35., GRID), (0.0185, 35., WINDOWS), (0.0186, -35., GRID), (0.001, 35., WINDOWS),
    (1.0, 0.62, GRID), (1.0, 0.6, WINDOWS), (1.0, 0., WINDOWS)])
def test_float64_tiles_of_few_cells(d, inc, launches):
    """Tiles that span less than half a bin, whose facets would all add to the same cells."""
    assert route('f64', facet_dx=d, inc_angle=np.deg2rad(inc)) == launches


@pytest.mark.parametrize("binsize,d,inc,mixed,f64", [
    (2.725, 1.33, 35., GRID, GRID), (2.725, 1.34, 35., WINDOWS, WINDOWS), (2.725, 1.34, -35., WINDOWS, WINDOWS),
    (0.454, 0.22, 35., GRID, GRID), (0.227, 0.08, 35., GRID, GRID), (0.227, 0.081, 35., WINDOWS, GRID),
    (0.227, 0.11, -35., WINDOWS, GRID), (0.227, 0.112, 35., WINDOWS, WINDOWS), (0.1, 0.01, 35., WINDOWS, GRID)])
def test_room_for_the_waves(binsize, d, inc, mixed, f64):
    """Tiles that leave six bins on each side of the grid, in the mixed form 2.5 m at least; a
    negative incidence spans as many bins as a positive one."""
    kw = dict(binsize=binsize, facet_dx=d, inc_angle=np.deg2rad(inc))
    assert route(**kw) == mixed
    assert route('f64', **kw) == f64


@pytest.mark.parametrize("raw,lo,launches", [
    (1 << 40, 1 << 41, GRID), ((1 << 40) + 8, (1 << 41) + 8, GRID), ((1 << 40) + 4, 1 << 41, WINDOWS),
    (1 << 40, (1 << 41) + 4, WINDOWS)])
def test_rows_off_their_pair_alignment(raw, lo, launches):
    """The fine grid folds the compensation row by complex64 vectors; rows aligned to a float only
    (never launched here) have to take the windows, which go by floats."""
    assert route(raw_d=raw, raw_lo_d=lo) == launches


@pytest.mark.gpu
@pytest.mark.parametrize("d", [1.0, 0.05, 0.005])
def test_sums_of_equal_facets(tmp_path, d):
    """A flat sea of equal, phaseless facets, whose float32 sums round the same way at every add, in
    tiles of some 38 rows where nothing bounds them.  Bar of a mixed bin against the float64 one:
    twice what the register windows come to here (1.4e-7 of the largest bin)."""
    pytest.importorskip("torch")
    from oceansar_b200.radarsim.sar_raw_nompi import RawGenerator
    from test_gpu_pulse_forms import make_cfg
    cfg = make_cfg(tmp_path, 2048, 2048, d, 35.0, 'vv', 1, 0, False)
    gens = [RawGenerator(cfg, precision=p, seed=3, overrides=dict(az_steps=8)) for p in ('f64', 'mixed')]
    for value in (1.1 - 0.7j, 1.3 - 1.9j, 0.3337 - 0.771j):
        raws = []
        for g in gens:
            for f in ('Dx', 'Dy', 'Dz', 'Diffx', 'Diffy'):
                g.surface.field(f).zero_()
            for r in (g.rndscat_m, g.rndscat_p):
                r.device()[0].fill_(value)
                if g.precision == 'mixed':
                    r.device32().fill_(value)
            g.reset()
            g._scat_d.fill_(1.0)
            g.t_last_rcs_bragg = 1e9                # no refresh: the planes stay as filled
            g.desc.k0 = 1e-12
            g.pulse(3, update_surface=False)
            raws.append(g.raw()[0, 0, 3])
        assert np.abs(raws[0]).max() > 100
        assert np.abs(raws[1] - raws[0]).max() <= 2.8e-7 * np.abs(raws[0]).max()
