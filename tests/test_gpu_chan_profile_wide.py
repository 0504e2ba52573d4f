"""Flattened lists that span more bins than the accumulation's fine grid: parts that go tap by tap
from the start, after their first facets, or by further windows; both element types, against the
oracle's sum.  Bars: float64 1e-12 (as the other orders); complex64 outputs take at most one
float32 add per CTA and bin, 148 x 2^-24 < 9e-6."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import range_profile as orp  # noqa: E402
from oceansar_b200 import _capi, _device  # noqa: E402
from oceansar_b200.radarsim import range_profile as rp  # noqa: E402

BS = 2.725


def bins_of(order, n, nbins, rs):
    """Bin positions of the facets."""
    part = -(-n // min(148, -(-n // 1024)))     # facets of a CTA's part
    i = np.arange(n)
    if order == "random":
        return rs.rand(n) * nbins * 1.1 - 0.05 * nbins
    if order == "rows":
        return (i % 1733) * (nbins * 0.97 / 1733) + rs.rand(n)
    late = (i % part) >= 4096
    if order == "late_far":                     # window 0 in the middle, the rest on both sides
        return np.where(late, rs.rand(n) * nbins, 0.5 * nbins + 20 * rs.rand(n))
    return np.where(late, 30 + 700 * rs.rand(n), 10 + 20 * rs.rand(n))      # late_near: one more window


@pytest.mark.parametrize("precision", ["f64", "c64"])
@pytest.mark.parametrize("order", ["random", "rows", "late_far", "late_near"])
@pytest.mark.parametrize("n,taps,ovs,nbins", [(1, 8, 20, 700), (5000, 7, 10, 700), (200001, 8, 20, 4000),
                                              (1000003, 16, 10, 12288), (700000, 8, 40, 3000)])
def test_wide_lists(precision, order, n, taps, ovs, nbins):
    rs = np.random.RandomState(n % 91)
    srg = bins_of(order, n, nbins, rs) * BS - BS
    scene = rs.randn(n) + 1j * rs.randn(n)
    if precision == "c64":
        scene = scene.astype(np.complex64).astype(np.complex128)
    bad = rs.permutation(n)[:2] if n > 1 else np.zeros(0, int)
    scene[bad[:1]] = complex(np.inf, 1.0)
    srg[bad[1:]] = np.nan
    sinc = rp.calc_sinc_vec(taps, ovs, Fs=1.1)
    ok = np.isfinite(srg) & np.isfinite(scene.real)
    ref = np.zeros(nbins, complex)
    orp.chan_profile(srg[ok], scene[ok], BS, -BS, sinc, taps, ovs, ref)
    hit = np.zeros(nbins, bool)
    for i in bad[:1]:
        b = int(np.floor((srg[i] + BS) / BS)) - taps // 2
        hit[max(0, b):max(0, min(nbins, b + taps))] = True
    if precision == "f64":
        out = np.zeros(nbins, complex)
        rp.chan_profile_numba(srg, scene, BS, -BS, sinc, taps, ovs, out)
    else:
        s_d, c_d = _device.to_device(srg, np.float64), _device.to_device(scene.astype(np.complex64), np.complex64)
        o_d, w_d = _device.zeros(nbins, np.complex64), _device.to_device(sinc, np.float32)
        _capi.call("ocs_chan_profile_c64", _device.ptr(s_d), _device.ptr(c_d), n, BS, -BS, _device.ptr(w_d), taps, ovs,
                   _device.ptr(o_d), nbins, _device.stream_ptr())
        out = o_d.cpu().numpy().astype(complex)
    assert (~np.isfinite(out) == hit).all()
    tol = 1e-12 if precision == "f64" else 9e-6
    assert np.linalg.norm((out - ref)[~hit]) <= tol * np.linalg.norm(ref[~hit])


@pytest.mark.parametrize("order", ["one_cell", "random"])
@pytest.mark.parametrize("n,ovs,nbins", [(600000, 20, 64), (3000001, 20, 512), (100000, 100, 40), (100000, 300, 40)])
def test_complex64_sums_of_many_equal_values(order, n, ovs, nbins):
    """Thousands of equal coefficients in one cell of the grid, whose float32 sum would round the same
    way at every add: the result keeps to the one float32 add per CTA and bin."""
    rs = np.random.RandomState(1)
    srg = BS * (7.3 + np.zeros(n) if order == "one_cell" else rs.rand(n) * nbins)
    sinc = rp.calc_sinc_vec(8, ovs, Fs=1.1)
    value = np.complex64(1.1 - 0.7j)
    ref = np.zeros(nbins, complex)
    orp.chan_profile(srg, np.full(n, complex(value)), BS, 0.0, sinc, 8, ovs, ref)
    s_d, c_d = _device.to_device(srg, np.float64), torch.full((n,), complex(value), dtype=torch.complex64, device="cuda")
    o_d, w_d = _device.zeros(nbins, np.complex64), _device.to_device(sinc, np.float32)
    _capi.call("ocs_chan_profile_c64", _device.ptr(s_d), _device.ptr(c_d), n, BS, 0.0, _device.ptr(w_d), 8, ovs,
               _device.ptr(o_d), nbins, _device.stream_ptr())
    out = o_d.cpu().numpy().astype(complex)
    assert np.abs(out - ref).max() <= 9e-6 * np.abs(ref).max()


@pytest.mark.parametrize("precision", ["f64", "c64"])
@pytest.mark.parametrize("n,nbins", [(70001, 700), (200001, 4000)])
def test_scene_off_its_pair_alignment(precision, n, nbins):
    """Scene values that start half a pair off the alignment of one vector load."""
    rs = np.random.RandomState(4)
    srg = rs.rand(n) * nbins * BS
    real = np.float64 if precision == "f64" else np.float32
    flat = rs.randn(2 * n + 1).astype(real)
    scene = flat[1:].astype(np.float64).view(np.complex128)
    sinc = rp.calc_sinc_vec(8, 20, Fs=1.1)
    ref = np.zeros(nbins, complex)
    orp.chan_profile(srg, scene, BS, 0.0, sinc, 8, 20, ref)
    s_d, f_d, w_d = (_device.to_device(a, t) for a, t in ((srg, np.float64), (flat, real), (sinc, np.float32)))
    o_d = _device.zeros(nbins, np.complex128 if precision == "f64" else np.complex64)
    _capi.call("ocs_chan_profile_" + precision, _device.ptr(s_d), f_d[1:].data_ptr(), n, BS, 0.0, _device.ptr(w_d), 8,
               20, _device.ptr(o_d), nbins, _device.stream_ptr())
    out = o_d.cpu().numpy().astype(complex)
    assert np.linalg.norm(out - ref) <= (1e-12 if precision == "f64" else 9e-6) * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [0, 1, 256, 1000, 1001, 2500])
def test_stored_tables(n):
    """Tables that one launch carries, exactly or not, and those that take several."""
    host = np.arange(n + 1, dtype=np.float32) * 0.37 - 5.0
    dst = torch.full((n + 8,), 9.0, dtype=torch.float32, device="cuda")
    _capi.call("ocs_store_table", _device.ptr(dst), host.ctypes.data, n, _device.stream_ptr())
    got = dst.cpu().numpy()
    np.testing.assert_array_equal(got[:n], host[:n])
    assert (got[n:] == 9.0).all()
