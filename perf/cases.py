"""The workloads the engine's speed is measured on: one pass each through the package's public calls.

A case is a detector of ``lumen_b200.detectors``, a source, a number of photons and the run's options. The detector and
its engine are kept, as a program that simulates keeps them; every pass is a whole call, from host inputs to host
results, at inputs (the source's place, the parameters' values, the run's seed) made from the case's seed.

    listed()              the cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   what a program holds before the call
    run(state)            the call and its outputs
    work(case)            the bytes and operations a pass cannot do without
    exact(case, seed)     the outputs that have a value without the simulation
"""

from __future__ import annotations

import functools

import numpy as np
import torch

from lumen_b200 import api, autograd, detectors, sources
from lumen_b200.readout import Axis, Grid, Group

# The kinds of run: photons from `lo` to `hi`, and steps a photon takes (measured, for the operations a pass needs).
KINDS = {
    "toy": dict(lo=1 << 12, hi=1 << 21, steps=1.0),
    "tank": dict(lo=1 << 16, hi=1 << 24, steps=2.8),
    "fit": dict(lo=1 << 16, hi=1 << 22, steps=2.9),
    "backward": dict(lo=1 << 16, hi=1 << 21, steps=5.6),
    "tracks": dict(lo=1 << 17, hi=1 << 23, steps=2.8),
    "lar": dict(lo=1 << 14, hi=1 << 17, steps=48.0),
    "readout": dict(lo=1 << 15, hi=1 << 20, steps=6.0),
    "solids": dict(lo=1 << 14, hi=1 << 17, steps=11.0),
    "panel64": dict(lo=1 << 16, hi=1 << 21, steps=2.0),
    "fog": dict(lo=1 << 14, hi=1 << 17, steps=47.0),
}

TANK_FIT = ("media/Water/absorption", "media/Water/rayleigh", "surfaces/BlackSheet/R",
            "surfaces/BlackSheet/sigma_alpha")  # fmt: skip
TRACK_FIT = ("media/Water/absorption", "media/Water/rayleigh", "surfaces/BlackSheet/R")
LAR_FIT = ("surfaces/CageSurface/R", "media/LAr/rayleigh")


def listed():
    return [
        # one vertex of an event-by-event study or one trial of an interactive session: the smallest call, all latency
        {"name": "toy_tank_4k", "kind": "toy", "photons": 4099},
        # the tutorial's run: the 8-PMT tank at 2^18 photons
        {"name": "toy_tank_256k", "kind": "toy", "photons": 1 << 18},
        # an ordinary run of the 2000-PMT water tank with 1 ns arrival-time histograms, a ragged number of photons
        {"name": "tank_1M", "kind": "tank", "photons": 1000003, "bins": 200},
        # the benchmark's own call, the largest: 2^24 photons of the same tank
        {"name": "tank_16M", "kind": "tank", "photons": 1 << 24, "bins": 200},
        # one iteration of a calibration fit: ground walls, the Jacobian in four parameters at values moved off a held
        # reference (common random numbers)
        {"name": "tank_fit_2M", "kind": "fit", "photons": 2000000, "gradients": 4, "held": True},
        # the same tank inside a torch optimiser: forward, then the adjoint's backward pass
        {"name": "tank_backward_1M", "kind": "backward", "photons": 1 << 20, "gradients": 3},
        # a batch of track events of uneven sizes, arrivals and their Jacobian per event
        {"name": "tracks_64_events_4M", "kind": "tracks", "photons": 4194301, "events": 64, "gradients": 3},
        # the liquid-argon box (booleans of boxes, multiple scattering): scintillation points with their Jacobian
        {"name": "lar_10000_points_128k", "kind": "lar", "photons": 131072, "events": 10000, "gradients": 2},
        # readout histograms (charge axes, delay cells, time grids) of a scintillator with Mie and WLS channels
        {"name": "readout_groups_300k", "kind": "readout", "photons": 300007},
        # every solid of the catalogue, tori among them
        {"name": "solids_box_100k", "kind": "solids", "photons": 100003},
        # a 3 um coating: the float64 navigator
        {"name": "coated_panel_f64_1M", "kind": "panel64", "photons": 1 << 20},
        # a strongly scattering medium (the diffusion jump), photons from explicit rows on the host
        {"name": "fog_rows_64k", "kind": "fog", "photons": 65537},
    ]


def draw(rng):
    kind = rng.choice(sorted(KINDS))
    k = KINDS[kind]
    n = int(round(k["lo"] * (k["hi"] / k["lo"]) ** rng.random()))
    case = {"kind": kind, "photons": min(n | (rng.random() < 0.5), k["hi"])}
    if kind == "tank":
        case["bins"] = rng.choice([0, 50, 200, 333])
    if kind in ("fit", "backward", "tracks", "lar"):
        case["gradients"] = rng.randint(1, {"fit": 4, "backward": 3, "tracks": 3, "lar": 2}[kind])
    if kind == "fit":
        case["held"] = rng.random() < 0.5
    if kind == "tracks":
        case["events"] = int(round(256 ** rng.random()))
    if kind == "lar":
        case["events"] = int(round(10000 ** rng.random()))
    return case


@functools.lru_cache(maxsize=None)
def _detector(kind):
    """The detector of a kind of run, built once: what a program loads at its start."""
    if kind == "toy":
        return detectors.toy_tank()
    if kind in ("tank", "backward", "tracks"):
        return detectors.cylinder_tank()
    if kind == "fit":
        return detectors.cylinder_tank(wall_finish="ground", sigma_alpha=0.1)
    if kind == "lar":
        return detectors.lar_box(sigma_alpha=0.1)
    if kind == "readout":
        return detectors.readout_tank()
    if kind == "solids":
        return detectors.solids_box()
    if kind == "panel64":
        return detectors.coated_panel(precision="float64")
    return detectors.fog_box()


def _in_tank(rng, n):
    """n points uniform in the tank's inner volume."""
    r, ph = 4.7 * np.sqrt(rng.uniform(size=n)), rng.uniform(0.0, 2.0 * np.pi, n)
    return np.stack([r * np.cos(ph), r * np.sin(ph), rng.uniform(-4.7, 4.7, n)], 1)


def _directions(rng, n):
    u = rng.normal(size=(n, 3))
    return u / np.linalg.norm(u, axis=1, keepdims=True)


def _counts(rng, total, events, spread=3.0):
    """`total` photons over `events`, uneven by up to 10^spread, each at least one."""
    share = 10.0 ** rng.uniform(0.0, spread, events)
    c = 1 + np.floor(share / share.sum() * (total - events)).astype(np.int64)
    c[np.argmax(c)] += total - c.sum()
    return c


def _values(det, names, rng, by=0.02):
    """The parameters `names` moved by a few per cent, as an optimiser moves them."""
    now = det.params()
    return {k: float(np.float32(np.ravel(now[k][1])[0] * (1.0 + by * rng.uniform(-1.0, 1.0)))) for k in names}


def prepare(case, seed):
    kind, n = case["kind"], int(case["photons"])
    det = _detector(kind)
    rng = np.random.default_rng([int(seed), n])
    api._engine(det)  # the detector is on the GPU before the call
    st = {"kind": kind, "det": det, "call": {"samples": n, "seed": int(rng.integers(1 << 30))}, "weight": 1.0}
    call = st["call"]
    if kind == "toy":
        st["weight"] = 2.0e5
        st["source"] = sources.Point(position=rng.uniform(-0.35, 0.35, 3), n_photons=2.0e5, lam=400.0)
        st["values"] = _values(det, ("surfaces/CathodeSurface/eff",), rng, 0.0)
    elif kind in ("tank", "fit", "backward"):
        st["source"] = sources.Point(position=_in_tank(rng, 1)[0], n_photons=1.0, lam_range=(300.0, 600.0))
        names = list(TANK_FIT if kind == "fit" else TRACK_FIT)[: int(case.get("gradients", 0))]
        if kind == "tank" and case.get("bins"):
            call["time_bins"] = (int(case["bins"]), 0.0, 200.0 / int(case["bins"]))
        if kind == "fit":
            st["values"] = _values(det, names, rng)
            call["gradients"] = names
            if case.get("held"):
                call["reference"] = _values(det, names, rng, 0.0)
        if kind == "backward":
            st["names"] = names
            st["x"] = torch.tensor(list(_values(det, names, rng).values()), dtype=torch.float64)
            st["cotangent"] = torch.from_numpy(rng.normal(size=det.n_sensor)).cuda()
    elif kind == "tracks":
        e = int(case["events"])
        u = _directions(rng, e)
        cnt = _counts(rng, n, e)
        st["source"] = sources.Tracks(start=0.7 * _in_tank(rng, e), direction=u, length=rng.uniform(0.3, 1.2, e),
                                      n_photons=cnt.astype(np.float64), lam_range=(300.0, 600.0), counts_=cnt)  # fmt: skip
        st["weight"] = float(n)
        call["gradients"] = list(TRACK_FIT)[: int(case["gradients"])]
    elif kind == "lar":
        e = min(int(case["events"]), n)
        st["source"] = sources.Scintillation(position=rng.uniform([-2.4, -1.9, -1.9], [2.4, 1.9, 1.9], (e, 3)),
                                             lam=128.0, tau=(6.0, 1500.0), fraction=0.25, n_photons=1.0)  # fmt: skip
        st["weight"] = float(e)
        call["gradients"] = list(LAR_FIT)[: int(case["gradients"])]
    elif kind == "readout":
        grid = Grid(axes=(Axis("wavelength", "wavelength", knots=(300.0, 350.0, 400.0, 450.0, 500.0, 550.0)),
                          Axis("theta", "theta", knots=(0.0, 0.5, 1.0, 1.6))),
                    delay_axes=(Axis("inc", "cos_incidence", edges=(0.0, 0.5, 1.0)),), t0=-2.0, dt=0.5, nt=60,
                    weighted=True, normalise=True)  # fmt: skip
        bands = Grid(axes=(Axis("gen", "generation", edges=(-0.5, 0.5, 1.5, 9.5)),), nt=40, t0=0.0, dt=1.0)
        call["groups"] = {"pmt": Group(grid, tuple(det.groups["pmt"]), rng.uniform(0.1, 0.3, grid.shape)), "ref": bands}
        st["source"] = sources.Point(position=rng.uniform(-0.3, 0.3, 3), n_photons=1.0, lam_range=(330.0, 480.0))
    elif kind == "solids":
        st["source"] = sources.Point(position=(*rng.uniform(-1.0, 1.0, 2), rng.uniform(-0.9, -0.6)), n_photons=1.0,
                                     lam=420.0)  # fmt: skip
    elif kind == "panel64":
        st["source"] = sources.Point(position=rng.uniform([3.0, -0.5, -0.5], [4.5, 0.5, 0.5]), n_photons=1.0, lam=420.0)
    else:
        st["source"] = sources.FromArrays(x=np.array([-1.5, 0.5, 0.0]) + rng.normal(0.0, 0.5, (n, 3)),
                                          d=_directions(rng, n), t=0.0, lam=rng.uniform(380.0, 450.0, n), w=1.0)  # fmt: skip
        st["weight"] = float(n)
        del call["samples"]
    return st


def _outputs(light):
    h = light.health
    out = {"arrivals": light.arrivals, "error": light.arrivals_error, "time": light.mean_arrival_time,
           "start": np.float64(h.start), "fates": np.array([getattr(h, k) for k in h.FATES]),
           "counts": np.array([h.photons, h.steps, h.records, h.nonfinite], np.int64)}  # fmt: skip
    if light.gradients is not None:
        out["gradients"] = {k.replace("/", "_"): v for k, v in light.gradients.items()}
    if light.diagnostics is not None:
        out["histogram"] = light.diagnostics["time"]
    for name, g in (light.groups or {}).items():
        out[name] = {k: v for k in ("charge", "charge2", "time", "late", "early", "pe_error")
                     if (v := getattr(g, k)) is not None}  # fmt: skip
    return out


def run(state):
    if state["kind"] == "backward":
        x = state["x"].clone().requires_grad_(True)
        arrivals = autograd.simulate(state["det"], state["source"], x, state["names"], **state["call"])
        arrivals.backward(state["cotangent"])
        return {"arrivals": arrivals.detach(), "gradient": x.grad}
    return _outputs(api.simulate(state["det"], state["source"], state.get("values"), **state["call"]))


# A step's operations: its random numbers (about 8 blocks of 20 rounds), one query of the geometry (about 40 box tests
# and 2 solids) and the surface's or medium's optics; each parameter's tangent adds about a tenth.
STEP_OPS = 3000


def work(case):
    kind, n = case["kind"], int(case["photons"])
    det = _detector(kind)
    sensors, events, grads = det.n_sensor, int(case.get("events", 1)), int(case.get("gradients", 0))
    scene = sum(v.nbytes for k, v in det.arrays.items() if isinstance(v, np.ndarray)) + np.asarray(det.pool).nbytes
    cells = events * sensors * (3 + int(case.get("bins", 0)) + grads)
    rows = n * 15 * 4 if kind == "fog" else events * 64
    return {"bytes": float(scene + rows + 8 * cells),
            "flops": float(n * KINDS[kind]["steps"] * STEP_OPS * (1.0 + 0.1 * grads))}  # fmt: skip


def exact(case, seed):
    """The start weights' sum (each event's photons share its weight, rounded to float32 a photon). Every other output
    is an estimate from random paths: it has no value of its own."""
    kind, n = case["kind"], int(case["photons"])
    if kind == "backward":
        return None
    if kind in ("toy", "tank", "fit", "readout", "solids", "panel64"):
        start = float(np.float32((2.0e5 if kind == "toy" else 1.0) / n)) * n
    elif kind == "lar":
        e = min(int(case["events"]), n)
        cnt = np.full(e, n // e, np.int64)
        cnt[: n - cnt.sum()] += 1
        start = float((np.float64(np.float32(1.0 / cnt)) * cnt).sum())
    else:
        start = float(n)
    return {"start": np.float64(start)}
