"""``chan_profile_numba(stream=S)``: every temporary belongs to S, and S comes after the work
pending on the caller's stream.  On the CPU against a recording stand-in for the stream calls; on
the GPU with work pending on the current stream that writes the inputs and a freed block."""
import contextlib

import numpy as np
import pytest
import torch

from oceansar_b200 import _capi, _device
from oceansar_b200.radarsim import range_profile as rp


class FakeStream(object):
    def __init__(self, handle):
        self.cuda_stream = handle
        self.after = []

    def wait_stream(self, other):
        self.after.append(other)


@pytest.mark.parametrize("handle_only", [False, True], ids=["stream", "handle"])
def test_temporaries_belong_to_the_given_stream(monkeypatch, handle_only):
    main, side = FakeStream(11), FakeStream(22)
    current = [main]
    log = []

    @contextlib.contextmanager
    def use(s):
        current.append(s)
        yield
        current.pop()

    monkeypatch.setattr(torch.cuda, "Stream", FakeStream)
    monkeypatch.setattr(torch.cuda, "ExternalStream", lambda h: side if h == 22 else None)
    monkeypatch.setattr(torch.cuda, "stream", use)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: current[-1])
    monkeypatch.setattr(_device, "require_cuda", lambda: torch.device("cpu"))
    empty, copy = _device.empty, _device.to_device
    monkeypatch.setattr(_device, "empty", lambda *a: (log.append(("alloc", current[-1], None)), empty(*a))[1])
    monkeypatch.setattr(_device, "to_device", lambda *a: (log.append(("copy", current[-1], None)), copy(*a))[1])
    monkeypatch.setattr(_capi, "call", lambda name, *a: log.append((name, current[-1], a[-1].value)))
    given = type("Handle", (), {"cuda_stream": 22})() if handle_only else side
    rp.chan_profile_numba(np.zeros(3), np.zeros(3, complex), 1.0, 0.0, rp.calc_sinc_vec(8, 20), 8, 20,
                          np.zeros(8, complex), stream=given)
    assert side.after == [main] and current == [main]
    assert {what for what, _, _ in log} == {"alloc", "copy", "ocs_store_table", "ocs_chan_profile_f64"}
    assert all(s is side for _, s, _ in log)
    assert all(h in (None, 22) for _, _, h in log)


@pytest.mark.gpu
def test_side_stream_after_pending_work():
    from oracle import range_profile as orp
    n, nbins = 5000, 300
    rs = np.random.RandomState(2)
    srg, scene = rs.rand(n) * 800.0, rs.randn(n) + 1j * rs.randn(n)
    sinc = rp.calc_sinc_vec(8, 20, Fs=1.1)
    ref = np.zeros(nbins, complex)
    orp.chan_profile(srg, scene, 2.725, 0.0, sinc, 8, 20, ref)
    side = torch.cuda.Stream()
    srg_h, scene_h = torch.from_numpy(srg).pin_memory(), torch.from_numpy(scene).pin_memory()
    srg_d = torch.zeros(n, dtype=torch.float64, device="cuda")
    scene_d = torch.zeros(n, dtype=torch.complex128, device="cuda")
    outs = [torch.zeros(nbins, dtype=torch.complex128, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    for out in outs:
        torch.cuda._sleep(20_000_000)               # some 10 ms of pending work, then the inputs
        srg_d.copy_(srg_h, non_blocking=True)
        scene_d.copy_(scene_h, non_blocking=True)
        block = torch.empty(161, dtype=torch.float32, device="cuda")
        torch.cuda._sleep(2_000_000)
        block.fill_(7.0)                            # pending on a block that is free from here on
        del block
        rp.chan_profile_numba(srg_d, scene_d, 2.725, 0.0, sinc, 8, 20, out, stream=side)
    torch.cuda.synchronize()
    for out in outs:
        assert np.linalg.norm(out.cpu().numpy() - ref) <= 1e-10 * np.linalg.norm(ref)
