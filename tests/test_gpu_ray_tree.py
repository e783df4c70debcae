"""The ray traversal's own tree (scene_create's node records) and the booleans' truth tables on the GPU against the
checker, which scans every candidate and runs the postfix programs: the same queries bit for bit at the sizes where a
tree or a table can go wrong. Exact: the engine's arithmetic is the checker's."""

import numpy as np
import pytest

import oracle
from lumen_b200 import detector as D
from lumen_b200 import geometry as G
from lumen_b200 import optics as O

pytestmark = pytest.mark.gpu


def _det(place, lv=None):
    water, glass = O.Material("Water", rindex=1.33), O.Material("Glass", rindex=1.5)
    box = G.Volume("Box", G.Box(2.0, 2.0, 2.0), "Water")
    place(box)
    return D.build(box, {"Water": water, "Glass": glass})


def _same(det, n=6000, seed=3):
    from lumen_b200 import make
    from lumen_b200.engine import Engine

    make.build()
    rng = np.random.default_rng(seed)
    o = rng.uniform(-1.99, 1.99, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d[: n // 8, 1] = 0.0  # rays along the boxes' planes
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    eng = Engine(det)
    gi, gf = (v.cpu().numpy() for v in eng.query(o, d))
    oi, of = oracle.query(det, o, d)
    assert (gi == oi).all(), np.flatnonzero((gi != oi).any(1))[:10]
    assert (gf.view(np.uint32) == of.view(np.uint32)).all()
    assert (eng.locate(o).cpu().numpy() == oracle.locate(det, o)).all()
    # the run's own traversal (the wavefront's and the persistent loop's node records): photon by photon
    from lumen_b200 import _abi as A
    from lumen_b200 import sources
    from lumen_b200.engine import DeviceSource, DeviceTallies

    src = sources.Point(position=(0.013, -0.021, 1.9), n_photons=1.0, lam=400.0)
    for variant in (0, 3):
        c = A.controls(variant=variant, max_vertices=64)
        ds = DeviceSource(src, 4096)
        T = DeviceTallies(det.n_sensor, 1, 0, 0.0, 1.0, 0)
        eng.trace((0, 1), 4096, source=ds, controls=c, tallies=T)
        R, _ = oracle.trace(det, (0, 1), 4096, source=src, samples=4096, controls=c)
        assert (T.counts.cpu().numpy()[:4] == R.counts[:4]).all()
        np.testing.assert_allclose(T.health.cpu().numpy(), R.health, rtol=1e-9, atol=1e-9)


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
