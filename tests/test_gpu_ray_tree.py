"""The ray traversal's own tree (scene_create's node records) and the booleans' truth tables on the GPU against the
checker, which scans every candidate and runs the postfix programs: the same photons' arrivals and the same queries bit
for bit at the sizes where a tree or a table can go wrong. Exact: the engine's arithmetic is the checker's."""

import numpy as np
import pytest

import oracle
from lumen_b200 import _abi as A
from lumen_b200 import detector as D
from lumen_b200 import detectors, sources
from lumen_b200 import geometry as G
from lumen_b200 import optics as O

pytestmark = pytest.mark.gpu


def _det(place):
    """A water box with what ``place`` puts in it: every placement a sensor that reflects 0.4 of the light and detects the
    rest's half, so that a photon's arrivals tell which surfaces it met, and when."""
    water, glass = O.Material("Water", rindex=1.33), O.Material("Glass", rindex=1.5)
    box = G.Volume("Box", G.Box(2.0, 2.0, 2.0), "Water")
    place(box)
    surf = O.OpticalSurface("Skin", "dielectric_metal", "polished", reflectivity=0.4, efficiency=0.5)
    names = [p.name for p in box.daughters]
    return D.build(box, {"Water": water, "Glass": glass}, borders=[("Box", k, surf) for k in names],
                   sensors={lv: lv for lv in sorted({p.volume.name for p in box.daughters})})  # fmt: skip


def _rays(n, half, seed):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-half, half, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d[: n // 8, 1] = 0.0  # rays along the boxes' planes
    return o, (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def _engine(det):
    from lumen_b200 import make
    from lumen_b200.engine import Engine

    make.build()
    return Engine(det)


def _traced(det, eng, half, n=1 << 15, seed=5):
    """The run's own traversal, the node records in the scene's own instantiation, in the wavefront's query kernel and in
    the persistent loop: each photon from its own place, its own event, so that every photon's arrivals and their times
    are compared (a photon's sums are made in its own order: exact)."""
    from lumen_b200.engine import DeviceRows, DeviceTallies

    o, d = _rays(n, half, seed)
    rows = sources.FromArrays(x=o, d=d, lam=400.0, event=np.arange(n)).rows()
    for variant in (0, A.VARIANT_WAVEFRONT):
        c = A.controls(variant=variant, max_vertices=64)
        T = DeviceTallies(det.n_sensor, n, 0, 0.0, 1.0, 0)
        eng.trace((0, 1), n, rows=DeviceRows(rows, eng.device), controls=c, tallies=T)
        rounds = variant == A.VARIANT_WAVEFRONT  # the fill, at least two rounds of two kernels, the drain, the moments
        assert eng.launches >= 7 if rounds else eng.launches <= 3, eng.launches
        R, _ = oracle.trace(det, (0, 1), n, rows=rows, controls=c, n_events=n)
        for k in ("arrival", "arrival_t"):
            got, want = getattr(T, k).cpu().numpy().reshape(n, -1), getattr(R, k).reshape(n, -1)
            bad = np.flatnonzero((got != want).any(1))
            assert len(bad) == 0, (k, len(bad), bad[:5], got[bad[:2]], want[bad[:2]])
        assert (T.counts.cpu().numpy()[:4] == R.counts[:4]).all()
        np.testing.assert_allclose(T.health.cpu().numpy(), R.health, rtol=1e-9, atol=1e-9)
    return R


def _same(det, n=6000, seed=3):
    """The navigator's entry points (every geometry's instantiation, which walks the scene's own nodes; the booleans'
    truth tables), then the run's traversal."""
    eng = _engine(det)
    o, d = _rays(n, 1.99, seed)
    gi, gf = (v.cpu().numpy() for v in eng.query(o, d))
    oi, of = oracle.query(det, o, d)
    assert (gi == oi).all(), np.flatnonzero((gi != oi).any(1))[:10]
    assert (gf.view(np.uint32) == of.view(np.uint32)).all()
    assert (eng.locate(o).cpu().numpy() == oracle.locate(det, o)).all()
    R = _traced(det, eng, 1.99)
    assert det.n_sensor == 0 or R.arrival.sum() > 0.0


@pytest.mark.parametrize("n", [0, 1, 2, 3, 33])
def test_few_items(n):
    """No node, a leaf as the root, one split, an odd tree."""
    rng = np.random.default_rng(n)

    def place(box):
        for k in range(n):
            at = (-1.7 + 0.56 * (k % 7), -1.6 + 0.6 * (k // 7), rng.uniform(-1.5, 1.5))
            box.place(G.Volume("B", G.Box(0.2, 0.15, 0.1), "Glass"), at, name=f"B{k}", copy=k)

    _same(_det(place))


def test_sizes_over_many_decades():
    """Items whose sizes and distances halve along a diagonal: a greedy split peels one item a level, past the
    traversal's stack, unless the tree is held to it."""

    def place(box):
        for k in range(40):
            s = 1.2 * 0.72**k
            box.place(G.Volume(f"B{k}", G.Box(0.1 * s, 0.1 * s, 0.1 * s), "Glass"), (s, s, s), name=f"B{k}", copy=k)

    _same(_det(place))


def test_equal_centres():
    """Nested shells share one centre: no axis orders them."""

    def place(box):
        for k in range(12):
            outer, inner = 1.6 - 0.1 * k, 1.57 - 0.1 * k
            box.place(G.Volume(f"S{k}", G.SphereShell(outer, inner), "Glass"), (0.0, 0.0, 0.0), name=f"S{k}", copy=k)

    _same(_det(place))


@pytest.mark.parametrize("ops", ["u", "s", "i", "sus", "susisu", "uuuuuuu", "sisusis"])
def test_booleans(ops):
    """Chains of 2 to 8 leaves (the table's last bit among them)."""
    rng = np.random.default_rng(len(ops))
    solid = G.Box(1.0, 0.9, 0.8)
    for k, o in enumerate(ops):
        part = G.Orb(0.6 + 0.04 * k) if k % 2 else G.Box(0.5, 1.1, 0.3 + 0.05 * k)
        kind = {"u": "union", "s": "subtraction", "i": "intersection"}[o]
        solid = G.Boolean(kind, solid, part, pos=tuple(rng.uniform(-0.5, 0.5, 3)))

    _same(_det(lambda box: box.place(G.Volume("Part", solid, "Glass"), (0.1, -0.2, 0.05), name="Part")))


@pytest.mark.parametrize("name,half", [("solids_box", 1.4), ("protrusion_box", 0.9), ("mesh_tank", 0.9)])
def test_extended_geometry(name, half):
    """Tori, clips and mesh chunks: the extended instantiation's walk over the records."""
    det = getattr(detectors, name)()
    R = _traced(det, _engine(det), half, n=1 << 14)
    assert R.arrival.sum() > 0.0
