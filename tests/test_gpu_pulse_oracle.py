"""Pulses in both accumulation forms (fine grid, register windows) and both precisions, stage-wise on
the same surface fields, with facets raised or sunk so far that they fall outside their tile's bins
and, on the last pulse, facets without a finite value, which must leave exactly their own bins
without one.  Bars over the finite bins: float64 against the oracle 1e-10, mixed against the oracle
1e-4 (those of the stage-wise parity tests; natural seas, as a facet 200 m up has its mixed phase to
3e-3 only); the two mixed forms, which differ in their sums alone, 96 x 2^-24 < 6e-6."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oceansar_b200.radarsim.sar_raw_nompi import RawGenerator  # noqa: E402
from oracle.sar_raw import SarRawSim  # noqa: E402
from test_gpu_pulse_forms import make_cfg  # noqa: E402

STEPS = [1, 2, 3]                               # 1: the Bragg refresh; 3: values that are not finite
NARROW = [(256, 70, 1.0, 'vv', 1, 0, True), (140, 35, 1.0, 'DP', 2, 0, True), (252, 20, 1.0, 'hh', 3, 1.5, True),
          (128, 64, 0.5, 'vv', 2, 0, False)]
WIDE = [(256, 70, 6.0, 'vv', 1, 0, True), (140, 35, 6.0, 'DP', 2, 0, True), (252, 20, 6.0, 'hh', 3, 1.5, True),
        (128, 64, 3.0, 'vv', 4, 0, False)]


def case(tmp_path, nx, ny, d, pol, num_ch, b_xti, spec):
    cfg = make_cfg(tmp_path, nx, ny, d, 35.0, pol, num_ch, b_xti, spec)
    text = open(cfg).read().split('\n')
    open(cfg, 'w').write('\n'.join('wh_tol=150.0' if t.split('=')[0].strip() == 'wh_tol' else t for t in text))
    return cfg


def raised(dz, seed):
    """A few per cent of the facets up to 220 m up or down."""
    rs = np.random.RandomState(seed)
    return np.where(rs.rand(*dz.shape) < 0.03, rs.uniform(-220., 220., dz.shape), dz).astype(np.float32)


def not_finite(ny, nx):
    return (0, 5, np.inf), (ny - 1, nx - 1, np.nan), (ny // 2, 77, np.inf)


def compare(got, ref, tol):
    fin = np.isfinite(ref)
    assert fin[:, :, :2].all() and not fin[:, :, 2].all() and fin[:, :, 2].any()
    np.testing.assert_array_equal(np.isfinite(got), fin)
    for k in range(3):
        r, g, m = ref[:, :, k], got[:, :, k], fin[:, :, k]
        assert np.linalg.norm((g - r)[m]) <= tol * np.linalg.norm(r[m])


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("scene", NARROW + WIDE)
def test_against_the_oracle(tmp_path, precision, scene):
    pol = scene[3]
    cfg = case(tmp_path, *scene)
    osim = SarRawSim(cfg, overrides=dict(az_steps=60), seed=3)
    gen = RawGenerator(cfg, precision=precision, overrides=dict(az_steps=60), seed=3)
    s = osim.surface
    s.set_t(0.1)
    osim.frozen = True                          # the fields stay as they are put
    if precision == 'f64':
        s.Dz = raised(s.Dz, scene[0])
    for f in gen.surface._fields:
        gen.surface.field(f).copy_(torch.from_numpy(np.ascontiguousarray(getattr(s, f))))
    pols = ('hh', 'vv') if pol == 'DP' else (pol,)
    for a in STEPS:
        if a == 3:
            for y, x, v in not_finite(s.Ny, s.Nx):
                for p, name in enumerate(pols):
                    getattr(osim, 'RCS_bragg_' + name)[0][y, x] = v
                    gen._scat_d.reshape(-1, 2, s.Ny, s.Nx)[p, 0, y, x] = v
        with np.errstate(invalid='ignore'):
            osim.pulse(a)
        gen.pulse(a, update_surface=False)
    ref = np.stack([getattr(osim, 'proc_raw_' + p) for p in pols])[:, :, STEPS]
    compare(gen.raw()[:, :, STEPS], ref, 1e-10 if precision == 'f64' else 1e-4)


@pytest.mark.parametrize("scene", NARROW)
def test_mixed_forms_agree(tmp_path, scene):
    """The register windows are reached by a series length that the fine grid does not address; the
    entries in use are those of the other pulse (start index plus pulse offset stay within two
    turns of the series, which the longer one holds)."""
    cfg = case(tmp_path, *scene)
    raws = []
    for length in (0, 2 ** 29):
        g = RawGenerator(cfg, precision='mixed', overrides=dict(az_steps=60), seed=3)
        if length:
            twice = [torch.cat([r.device32().reshape(-1)] * 2) for r in (g.rndscat_m, g.rndscat_p)]
            g.desc.s_m32_d, g.desc.s_p32_d = (t.data_ptr() for t in twice)
            assert all(r.tind(0.1) < len(t) // 2 for r, t in zip((g.rndscat_m, g.rndscat_p), twice))
            g.desc.n_m = g.desc.n_p = length
        s = g.surface
        s.set_t(0.1)
        dz = s.field('Dz')
        dz.copy_(torch.from_numpy(raised(dz.cpu().numpy(), scene[0])))
        for a in STEPS:
            if a == 3:
                for y, x, v in not_finite(s.Ny, s.Nx):
                    g._scat_d.reshape(-1, 2, s.Ny, s.Nx)[:, 0, y, x] = v
            g.pulse(a, update_surface=False)
        raws.append(g.raw()[:, :, STEPS])
    compare(raws[0], raws[1], 6e-6)
