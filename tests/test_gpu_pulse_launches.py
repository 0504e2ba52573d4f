"""The launch count that the pulse dispatch reports, against the routes' definitions: 60 pulses
with two Bragg refreshes, two surface passes and a pulse each; a row table for the
register-window kernels, which also take two float64 outputs at a time."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oceansar_b200.radarsim.sar_raw_nompi import RawGenerator  # noqa: E402
from test_gpu_pulse_forms import make_cfg  # noqa: E402


@pytest.mark.parametrize("precision,d,num_ch,pulse", [
    ('mixed', 1.0, 2, 1), ('mixed', 6.0, 2, 2),
    ('f64', 1.0, 4, 1), ('f64', 6.0, 4, 3),
])
def test_launches(tmp_path, precision, d, num_ch, pulse):
    cfg = make_cfg(tmp_path, 64, 32, d, 35.0, 'vv', num_ch, 0, True)
    g = RawGenerator(cfg, precision=precision, seed=3, overrides=dict(az_steps=60))
    assert g.kernel_launches_per_scene() == 60 * (2 + pulse) + 2
