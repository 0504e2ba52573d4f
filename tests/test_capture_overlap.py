"""``RawGenerator.capture``'s order of the scene: what the caller asks for, or the faster one.  On the
CPU with stand-ins for the stream calls and the pulses; on the GPU both orders, recorded or run,
against the plain loop."""
import contextlib
import os

import numpy as np
import pytest
import torch

from oceansar_b200.radarsim.sar_raw_nompi import RawGenerator

G = os.path.join(os.path.dirname(__file__), "golden")


class Surface(object):
    _aux = False

    def __init__(self, n):
        self.Nx = self.Ny = n


def generator(precision, n, npol=1, num_ch=1, balancer=None):
    g = object.__new__(RawGenerator)
    g.precision, g.surface, g.npol, g.num_ch = precision, Surface(n), npol, num_ch
    g.frozen, g.balancer, g.stream = False, balancer, None
    return g


@pytest.mark.parametrize("precision,n,npol,num_ch,pays", [
    ('mixed', 512, 1, 1, True), ('mixed', 1024, 1, 1, False), ('mixed', 1024, 1, 2, True),
    ('mixed', 2048, 2, 1, True), ('f64', 256, 1, 1, False), ('f64', 2048, 2, 4, False)])
@pytest.mark.parametrize("asked", [None, True, False])
@pytest.mark.parametrize("can", [True, False])
def test_order_of_a_captured_scene(monkeypatch, precision, n, npol, num_ch, pays, asked, can):
    class Stream(object):
        def wait_stream(self, other):
            pass

    for name, fake in (("Stream", Stream), ("current_stream", Stream), ("CUDAGraph", object),
                       ("synchronize", lambda: None), ("graph", lambda *a, **k: contextlib.nullcontext())):
        monkeypatch.setattr(torch.cuda, name, fake)
    g = generator(precision, n, npol, num_ch, None if can else object())
    ran = []
    g.reset = lambda: None
    g.run = lambda: ran.append('serial')
    g.run_overlapped = lambda: ran.append('overlapped')
    g._second_desc = lambda: None
    g.capture(**({} if asked is None else dict(overlap=asked)))
    want = can and (pays if asked is None else asked)
    assert ran == ['serial', 'overlapped' if want else 'serial']


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["c1small", "c3small", "c1lut"])
@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("how", ["run", "capture", "capture_serial"])
def test_orders_agree(name, precision, how):
    cfg = os.path.join(G, "cfg", name + ".cfg")
    a, b = (RawGenerator(cfg, precision=precision, seed=0) for _ in range(2))
    a.run()
    if how == "run":
        b.run_overlapped()
    else:
        b.capture(overlap=how == "capture")
        b.replay()
    torch.cuda.synchronize()
    assert (getattr(b, '_desc_b', None) is None) == (how == "capture_serial")
    tol = 1e-12 if precision == "f64" else 1e-5
    ref = a.raw()
    assert np.linalg.norm(b.raw() - ref) <= tol * np.linalg.norm(ref)
    np.testing.assert_allclose(b.nrcs_avg(), a.nrcs_avg(), rtol=tol)
