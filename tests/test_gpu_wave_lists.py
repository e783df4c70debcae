"""The wavefront over its lists of live slots, in every geometry and precision, against the persistent loop on the same
photons: the counts are equal and the FP64 sums agree to their order (rel 1e-9, absolute where a sum cancels); and a
run's results from its tallies (lumen_b200_finish) against the formulas in numpy, bit for bit."""

import numpy as np
import pytest
import torch

from lumen_b200 import _abi as A
from lumen_b200 import api, detectors, sources
from lumen_b200.engine import DeviceSource, DeviceTallies, Engine

pytestmark = pytest.mark.gpu

AT = {"toy_tank": (0.05, 0.02, 0.1), "solids_box": (0.05, 0.02, -0.6), "mesh_tank": (0.0, 0.5, -0.6),
      "wire_planes": (0.0, 0.1, 0.05), "protrusion_box": (0.1, -0.05, 0.6), "lar_box": (0.2, 0.3, 0.1),
      "coated_panel": (4.0, 0.1, 0.1), "readout_tank": (0.1, 0.0, 0.05)}  # fmt: skip
_engines = {}


def _engine(name, prec):
    if (name, prec) not in _engines:
        from lumen_b200 import make

        make.build()
        det = getattr(detectors, name)()
        _engines[name, prec] = Engine(det.with_precision(prec) if prec == "float64" else det)
    return _engines[name, prec]


def _run(eng, name, n, grads=(), **kw):
    det = eng.det
    src = sources.Point(position=AT[name], n_photons=1.0, lam=420.0)
    T = DeviceTallies(det.n_sensor, 1, 0, 0.0, 1.0, len(grads))
    c = A.controls(grad_tabs=[det.params_index[g] for g in grads], **kw)
    eng.trace((0, 5), n, source=DeviceSource(src, n), controls=c, tallies=T)
    if kw.get("variant") == A.VARIANT_WAVEFRONT and n >= 8192:  # the fill, two rounds or more, the drain, the moments
        assert eng.launches >= 7
    else:
        assert eng.launches <= 3
    return T


def _agree(a, b):
    assert (a.counts.cpu().numpy()[:4] == b.counts.cpu().numpy()[:4]).all()
    for k in ("arrival", "arrival_t", "arrival2", "health"):
        x, y = getattr(a, k).cpu().numpy(), getattr(b, k).cpu().numpy()
        np.testing.assert_allclose(x, y, rtol=1e-9, atol=1e-12, err_msg=k)
    if a.jac is not None:
        x, y = a.jac.cpu().numpy(), b.jac.cpu().numpy()
        np.testing.assert_allclose(x, y, rtol=1e-7, atol=1e-10)


@pytest.mark.parametrize("name", sorted(AT))
@pytest.mark.parametrize("prec", ["float32", "float64"])
@pytest.mark.parametrize("n", [1, 4099, 8192, 20011])
def test_every_scene(name, prec, n):
    """Below the rounds (the persistent loop alone), at their first size, and blocks with a part of one."""
    eng = _engine(name, prec)
    _agree(_run(eng, name, n, variant=A.VARIANT_WAVEFRONT), _run(eng, name, n, variant=0))


@pytest.mark.parametrize("name,prec", [("toy_tank", "float32"), ("protrusion_box", "float32"), ("coated_panel", "float64")])
@pytest.mark.parametrize("asynchronous", [False, True])
def test_refill(name, prec, asynchronous):
    """More photons than slots (2^16): the refill, its end inside a round, and with LUMEN_F_ASYNC a drain that resumes
    the slots and takes the photons left."""
    eng = _engine(name, prec)
    kw = dict(flags=A.F_ASYNC, wave_rounds=2) if asynchronous else {}
    n = 3 * (1 << 16) + 77
    a = _run(eng, name, n, variant=A.VARIANT_WAVEFRONT, wave_slots_log2=16, **kw)
    torch.cuda.synchronize()
    _agree(a, _run(eng, name, n, variant=0))


def test_tangents_with_clips_and_float64():
    for name, prec, grads in (("solids_box", "float32", ["media/Water/absorption", "surfaces/Wall/R"]),
                              ("coated_panel", "float64", ["media/Water/absorption"])):  # fmt: skip
        eng = _engine(name, prec)
        _agree(_run(eng, name, 9001, grads, variant=A.VARIANT_WAVEFRONT), _run(eng, name, 9001, grads, variant=0))


@pytest.mark.parametrize("name,grads", [("readout_tank", ()), ("protrusion_box", ()), ("mesh_tank", ("surfaces/Wall/R",))])
def test_largest_blocks(name, grads):
    """Enough live slots for the step's blocks of 512 (scenes with facets), the last one ragged; fewer as they end."""
    eng = _engine(name, "float32")
    _agree(_run(eng, name, 152001, grads, variant=A.VARIANT_WAVEFRONT), _run(eng, name, 152001, grads, variant=0))


def test_step_budget_ends_the_rounds():
    eng = _engine("lar_box", "float32")
    src = sources.Point(position=AT["lar_box"], n_photons=1.0, lam=420.0)
    T = DeviceTallies(eng.det.n_sensor)
    c = A.controls(variant=A.VARIANT_WAVEFRONT, step_budget=2000)
    with pytest.raises(A.StepBudgetExhausted):
        eng.trace((0, 5), 1 << 14, source=DeviceSource(src, 1 << 14), controls=c, tallies=T)
    assert int(T.counts[A.C_ABORTED]) == 1
    _agree(_run(eng, "lar_box", 9001, variant=A.VARIANT_WAVEFRONT), _run(eng, "lar_box", 9001, variant=0))  # serves the next


@pytest.mark.parametrize("events,sensors,bins,grads", [(1, 1, 0, 0), (1, 8, 3, 2), (5, 77, 0, 1), (300, 120, 7, 8)])
def test_results_are_numpys(events, sensors, bins, grads):
    eng = _engine("toy_tank", "float32")
    g = torch.Generator().manual_seed(events)
    T = DeviceTallies(sensors, events, bins, 0.0, 1.0, grads)
    x = torch.rand(events, sensors, generator=g, dtype=torch.float64)
    x[0, 0] = 0.0
    T.arrival.copy_(x)
    T.arrival_t.copy_(x * torch.rand(events, sensors, generator=g, dtype=torch.float64) * 90.0)
    T.arrival2.copy_(x * x * torch.rand(events, sensors, generator=g, dtype=torch.float64) * 2.0)
    want_bad = 0
    if sensors > 3:
        T.arrival2[0, 3] = float("nan")
        T.arrival[-1, 2] = float("inf")
        want_bad = 2
    if bins:
        T.hist[0, 0, 0] = float("-inf")
        want_bad += 1
    arr, t, x2 = (v.cpu().numpy().copy() for v in (T.arrival, T.arrival_t, T.arrival2))
    first = np.concatenate([[0], np.cumsum(np.arange(events) % 4)]).astype(np.int64)  # events of 0, 1, 2 and 3 photons
    n = 1000.0 if events == 1 else np.diff(first)[:, None]
    eng.finish(T, 1000, torch.from_numpy(first).cuda() if events > 1 else None)
    with np.errstate(all="ignore"):
        error = api.moment_error(x2, arr, n)
        time = np.where(arr > 0, t / np.where(arr > 0, arr, 1.0), np.nan)
    np.testing.assert_array_equal(T.arrival2.cpu().numpy(), error)
    np.testing.assert_array_equal(T.arrival_t.cpu().numpy(), time)
    assert int(T.nonfinite.item()) == want_bad


def test_results_of_a_tracer_on_the_device():
    """simulate_sharded with a caller's tracer whose tallies are on the GPU: the results of the engine's own share."""
    from lumen_b200 import distributed

    eng = _engine("toy_tank", "float32")
    det, src = eng.det, sources.Point(position=AT["toy_tank"], n_photons=1.0, lam=420.0)

    def tracer(first, n, key, controls, T):
        T = DeviceTallies(T.arrival.shape[1], T.arrival.shape[0], 0, 0.0, 1.0, 0)
        eng.trace(key, n, source=DeviceSource(src, 4099, det=det), first_id=first, controls=controls, tallies=T)
        return T

    want = distributed.simulate_sharded(det, src, samples=4099, seed=3)
    got = distributed.simulate_sharded(det, src, samples=4099, seed=3, tracer=tracer)
    for k in ("arrivals", "arrivals_error", "mean_arrival_time"):
        np.testing.assert_allclose(getattr(got, k), getattr(want, k), rtol=1e-9, atol=1e-12)
    assert got.health.photons == 4099
