"""Scene batches with scenes whose tiles the fine grid does not take (6 m facets; short tiles of
fine facets), beside fine-grid ones and after them in the same slot, against the scenes alone.
Bars: those of the batch (relative L2 of the raw cube 1e-5 mixed and 1e-12 float64, NRCS 1e-6 and
1e-12)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oceansar_b200 import _capi  # noqa: E402
from oceansar_b200.radarsim.batch import SceneBatch  # noqa: E402
from oceansar_b200.radarsim.sar_raw_nompi import RawGenerator  # noqa: E402
from test_gpu_pulse_forms import make_cfg  # noqa: E402

GRID, WIDE = 0, 2
# nx, ny, d, inc, pol, channels, b_xti, spec, tile rows, class of the mixed and of the float64 batch
SCENES = [(252, 70, 6.0, 35.0, 'vv', 2, 1.5, True, 0, WIDE, WIDE), (256, 128, 1.0, 35.0, 'DP', 2, 0, True, 0, GRID, GRID),
          (140, 63, 6.0, 35.0, 'DP', 2, 0, True, 32, WIDE, WIDE), (256, 128, 1.0, 20.0, 'vv', 3, 0, False, 128, WIDE, GRID),
          (256, 128, 1.0, 35.0, 'hh', 1, 0, True, 128, GRID, GRID), (128, 64, 6.0, 35.0, 'vv', 1, 0, False, 0, WIDE, WIDE)]


def check(gens, refs, precision):
    tol = (1e-5, 1e-6) if precision == 'mixed' else (1e-12, 1e-12)
    for g, (raw, nrcs) in zip(gens, refs):
        assert np.isfinite(raw).all() and np.abs(raw).max() > 0
        assert np.linalg.norm(g.raw() - raw) <= tol[0] * np.linalg.norm(raw)
        assert np.linalg.norm(g.nrcs_avg() - nrcs) <= tol[1] * np.linalg.norm(nrcs)


def alone(cfg, precision, seed):
    g = RawGenerator(cfg, precision=precision, seed=seed, overrides=dict(az_steps=60))
    g.run()
    return g.raw(), g.nrcs_avg()


def scenes(tmp_path, precision, which):
    cfgs, refs = [], []
    for k in which:
        (tmp_path / str(k)).mkdir()
        cfgs.append(make_cfg(tmp_path / str(k), *SCENES[k][:8]))
        refs.append(alone(cfgs[-1], precision, k))
    gens = [RawGenerator(c, precision=precision, seed=k, overrides=dict(az_steps=60)) for c, k in zip(cfgs, which)]
    return gens, refs


@pytest.mark.parametrize("precision", ["mixed", "f64"])
@pytest.mark.parametrize("graphs", [False, True])
def test_batch_of_both_classes(tmp_path, precision, graphs):
    gens, refs = scenes(tmp_path, precision, range(len(SCENES)))
    b = SceneBatch(max_slots=8, precision=precision)
    for g, s in zip(gens, SCENES):
        slot = b.add(g, tile_rows=s[8])
        assert _capi.load().ocs_batch_kind(b._h, slot) == s[9 if precision == 'mixed' else 10]
    assert _capi.load().ocs_batch_kind(b._h, 7) < 0
    b.run(pulse_block=16, use_graphs=graphs)
    torch.cuda.synchronize()
    check(gens, refs, precision)
    b.close()


@pytest.mark.parametrize("precision", ["mixed", "f64"])
@pytest.mark.parametrize("first", [6.0, 1.0])
def test_slot_of_another_class(tmp_path, precision, first):
    """Scenes of one size but of two classes, one after the other in the same slot: the steps
    recorded for the first must not be replayed for the second."""
    b = SceneBatch(max_slots=1, precision=precision)
    for k, d in enumerate((first, 7.0 - first, first)):
        (tmp_path / str(k)).mkdir()
        cfg = make_cfg(tmp_path / str(k), 128, 64, d, 35.0, 'vv', 1, 0, True)
        ref = alone(cfg, precision, k)
        g = RawGenerator(cfg, precision=precision, seed=k, overrides=dict(az_steps=60))
        b.add(g)
        b.run(pulse_block=15)
        torch.cuda.synchronize()
        check([g], [ref], precision)
    b.close()
