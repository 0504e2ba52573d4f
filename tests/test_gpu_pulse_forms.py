"""The split-range mixed pulse in both accumulation forms (fine grid / register windows), at the
edges of its tiles, and the Bragg refresh pass: raw rows and NRCS sums against the float64
form, stage-wise on the same surface fields (the float64 form is held to the oracle within
1e-10 elsewhere).  Bars: those of the mixed form (relative L2 1e-4)."""
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oceansar_b200.radarsim.sar_raw_nompi import RawGenerator  # noqa: E402

CFG = os.path.join(os.path.dirname(__file__), "golden", "cfg", "c1small.cfg")


def make_cfg(tmp_path, nx, ny, d, inc, pol, num_ch, b_xti, spec=True):
    text = open(CFG).read()
    for key, val in (('Lx', nx * d), ('Ly', ny * d), ('dx', d), ('dy', d), ('opt_res', False), ('inc_angle', inc),
                     ('pol', pol), ('num_ch', num_ch), ('b_ati', '5.0' if num_ch > 1 else '0'), ('b_xti', b_xti),
                     ('scat_spec_enable', spec), ('spread_model', 'cos2s'), ('wind_U', 6.0)):
        lines = []
        for line in text.split('\n'):
            lines.append('%s=%s' % (key, val) if line.split('=')[0].strip() == key else line)
        text = '\n'.join(lines)
    path = tmp_path / "case.cfg"
    path.write_text(text)
    return str(path)


# d = 1 m: a 128-column tile spans some 27 bins (fine grid); d = 6 m: some 160 (windows)
@pytest.mark.parametrize("nx,ny,d,inc,pol,num_ch,b_xti,spec", [
    (12, 10, 1.0, 35.0, 'vv', 1, 0, True),
    (128, 5, 1.0, 35.0, 'vv', 2, 0, True),
    (140, 63, 1.0, 35.0, 'hh', 3, 1.5, True),
    (252, 70, 1.0, 12.0, 'vv', 2, 0, True),
    (252, 70, 1.0, 35.0, 'DP', 2, 0, True),
    (256, 9, 0.5, 45.0, 'vv', 4, 1.0, False),
    (512, 640, 1.0, 25.0, 'vv', 2, 0, True),
    (140, 63, 6.0, 35.0, 'vv', 2, 1.5, True),
    (252, 20, 6.0, 35.0, 'DP', 2, 0, True),
    (256, 160, 3.0, 45.0, 'vv', 1, 0, False),
])
def test_mixed_against_f64(tmp_path, nx, ny, d, inc, pol, num_ch, b_xti, spec):
    cfg = make_cfg(tmp_path, nx, ny, d, inc, pol, num_ch, b_xti, spec)
    gens = [RawGenerator(cfg, precision=p, seed=3, overrides=dict(az_steps=60)) for p in ('f64', 'mixed')]
    steps = [0, 1, 52, 53]                      # 52: the second Bragg refresh (ocean dt 0.05 s, 1 kHz)
    for g in gens:
        g.surface.set_t(0.1)
        for a in steps:
            g.pulse(a, update_surface=False)
        assert g._refreshes == [0, 52]
    ref, got = gens[0].raw(), gens[1].raw()
    assert np.isfinite(ref).all() and np.abs(ref[:, :, steps]).max() > 0
    assert np.linalg.norm(got - ref) <= 1e-4 * np.linalg.norm(ref)
    for p in range(ref.shape[0]):
        for c in range(ref.shape[1]):
            for a in steps:
                assert np.linalg.norm(got[p, c, a] - ref[p, c, a]) <= 1e-4 * np.linalg.norm(ref[p, c, a])
    b64, b32 = (g.nrcs_bragg_d.cpu().numpy() for g in gens)
    assert np.allclose(b32, b64, rtol=1e-5, atol=0) and (b64[:, 52] > 0).all()
    s64, s32 = (g.nrcs_spec_d.cpu().numpy() for g in gens)
    assert np.allclose(s32, s64, rtol=1e-4, atol=1e-12)
