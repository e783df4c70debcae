"""The wavefront at the limits of what a call holds beside its tallies: its page-locked word over refused calls,
and the rounds of an asynchronous call after small synchronous ones."""

import ctypes

import numpy as np
import pytest
import torch

from lumen_b200 import _abi as A
from lumen_b200 import detectors, sources
from lumen_b200.engine import DeviceSource, DeviceTallies, Engine

pytestmark = pytest.mark.gpu


def _setup(name, at, n):
    from lumen_b200 import make

    make.build()
    det = getattr(detectors, name)()
    eng = Engine(det)
    src = sources.Point(position=at, n_photons=1.0, lam=420.0)
    return eng, DeviceSource(src, n), DeviceTallies(det.n_sensor)


def _resident_kb():
    for line in open("/proc/self/status"):
        if line.startswith("VmRSS"):
            return int(line.split()[1])
    raise RuntimeError("no VmRSS")


def test_refused_calls_keep_no_page_locked_memory():
    """A call refused before its first launch (more cells than the tallies' limit) gives its word back: 40,000 of them
    (at least 512 bytes of page-locked memory each, where each kept its own) leave the process its size."""
    eng, ds, T = _setup("toy_tank", (0.05, 0.02, 0.1), 1 << 14)
    c = A.controls(variant=A.VARIANT_WAVEFRONT)
    eng.trace((0, 1), 1 << 14, source=ds, controls=c, tallies=T)
    call = (eng.h, None, ctypes.byref(ds.c), 0, 1, 0, 1 << 14, ctypes.byref(c), ctypes.byref(T.c), None)
    events, T.c.n_events = T.c.n_events, 2**31 - 1
    assert T.arrival.shape[1] * T.c.n_events >= 2**32
    for _ in range(100):
        assert eng.lib.lumen_b200_trace(*call) == A.ERR_ARG
    before = _resident_kb()
    for _ in range(40000):
        eng.lib.lumen_b200_trace(*call)
    grown = _resident_kb() - before
    T.c.n_events = events
    T.zero_()
    eng.trace((0, 1), 1 << 14, source=ds, controls=c, tallies=T)
    assert int(T.counts[A.C_PHOTONS]) == 1 << 14
    assert grown < 4096, f"{grown} kB"


@pytest.mark.parametrize("n", [4096, 16384])
def test_rounds_of_an_asynchronous_call_after_a_small_one(n):
    """An asynchronous call takes its rounds from the scene's last synchronous wavefront call, a small one too (one the
    persistent loop ran, or whose rounds ended well before a 64th of its slots were live): the liquid-argon box's photons
    take some 48 steps each."""
    eng, ds, T = _setup("lar_box", (0.2, 0.3, 0.1), 1 << 16)
    eng.trace((0, 1), n, source=ds, controls=A.controls(variant=A.VARIANT_WAVEFRONT), tallies=T)
    steps = float(T.counts[A.C_STEPS]) / n
    assert steps > 20.0
    T.zero_()
    eng.trace((0, 1), 1 << 16, source=ds, tallies=T, controls=A.controls(variant=A.VARIANT_WAVEFRONT, flags=A.F_ASYNC))
    launches = eng.launches
    torch.cuda.synchronize()
    assert int(T.counts[A.C_PHOTONS]) == 1 << 16
    assert 2 * 1.5 * steps < launches < 2 * 5.0 * steps, (launches, steps)
    assert np.isfinite(T.health.cpu().numpy()).all()
