"""The order in which a step's binning leaves the particles: the stable sort of the
stored particles by cell key, against numpy's on the oracle's keys of the positions
before the step (whole numbers: equal), where the kernels' ways of ordering a block
end (768 and 4,096 particles in it, 128 in a cell, tiles of 4,096, 2^24 in the scene),
and far beyond."""
import numpy as np
import pytest

from oracle import oracle as O
from snow_gb300 import scenes

gpu = pytest.mark.gpu

# particles per (block, cell): {(block x, y, z): [particles of cell 0, 1, ...]}
CROWDS = {
    "block 768": {(2, 2, 2): [768]},
    "block 769": {(2, 2, 2): [769]},
    "cells 128": {(2, 2, 2): [128] * 7, (5, 2, 2): [128, 1, 640]},
    "cells 129": {(2, 2, 2): [129] + [128] * 6, (5, 2, 2): [0, 700, 129], (3, 5, 2): [40] * 64},
    "tiles": {(2, 2, 2): [64] * 64, (5, 2, 2): [64] * 63 + [65], (2, 5, 2): [128] * 64, (5, 5, 2): [8193]},
    "one cell": {(2, 2, 2): [20_000, 0, 1, 300], (6, 6, 6): [3]},
    "many blocks": {(x, y, 3): [0, 130 + 7 * x, 20, 500 * y] for x in range(1, 7) for y in range(1, 7)},
}


def _scene(crowd, seed):
    rng = np.random.default_rng(seed)
    s = scenes.unit_box_scene(32, young=1.0, dt=2e-3, name="crowd")
    at = [np.array([4 * b + c for b, c in zip(block, (k & 3, k >> 2 & 3, k >> 4))])
          for block, cells in crowd.items() for k, n in enumerate(cells) for _ in range(n)]
    s.x = ((np.array(at) + rng.uniform(0.02, 0.98, (len(at), 3))) * s.grid_spacing).astype(np.float32)
    s.x += np.asarray(s.grid_pos, np.float32)
    s.x = s.x[rng.permutation(len(at))]
    s.v = rng.uniform(-3.0, 3.0, s.x.shape).astype(np.float32)  # a fifth of a cell a step
    s.m = np.full(len(at), 1e-5, np.float32)
    return s


def _binned(order, x, s):
    """The order after a binning of particles stored in `order` (x in upload order)."""
    keys = O.cell_keys(x, s.grid_pos, s.grid_dim, s.grid_spacing)[1]
    return order[np.argsort(keys[order], kind="stable")]


@pytest.fixture(scope="module")
def ctx():
    from snow_gb300 import api
    return api.Context(0)


@gpu
@pytest.mark.parametrize("crowd", list(CROWDS))
def test_binning_is_the_stable_sort_by_cell(ctx, crowd):
    from snow_gb300 import api
    s = _scene(CROWDS[crowd], 71)
    g = api.SimScene(ctx, s, sort_interval=1).upload()
    order = np.arange(s.n, dtype=np.uint32)
    assert np.array_equal(g.storage_order(), order)
    order = _binned(order, s.x, s)
    assert np.array_equal(g.init().storage_order(), order)
    x = s.x
    for _ in range(4):
        before = g.phase_times()["binnings"]
        g.step(s.dt, 1)
        if g.phase_times()["binnings"] > before:
            order = _binned(order, x, s)
        assert np.array_equal(g.storage_order(), order)
        x = g.check().download()["x"]
    assert g.phase_times()["binnings"] >= 3
    g.close()


@gpu
def test_binning_of_more_than_two_to_the_24_particles(ctx):
    """Indices of five digits; half a million particles in one block, the others
    sixteen to a cell."""
    from snow_gb300 import api
    n, crowd = (1 << 24) + 5, 1 << 19
    rng = np.random.default_rng(76)
    s = scenes.unit_box_scene(128, young=1.0, dt=1e-4, name="crowd")
    s.x = rng.random((n, 3), dtype=np.float32) * np.float32(0.75) + np.float32(0.125)
    s.x[:crowd] = ((np.array([40, 44, 48]) + 4 * rng.random((crowd, 3))) * s.grid_spacing).astype(np.float32)
    s.x[:] = s.x[rng.permutation(n)]
    s.v = np.zeros_like(s.x)
    s.m = np.full(n, 1e-6, np.float32)
    g = api.SimScene(ctx, s).upload().init()
    assert np.array_equal(g.storage_order(), _binned(np.arange(n, dtype=np.uint32), s.x, s))
    g.close()


@gpu
def test_binning_of_a_batch_is_each_scenes_own(ctx):
    from snow_gb300 import api
    scs = [_scene(CROWDS[k], 72 + i) for i, k in enumerate(("one cell", "cells 128", "many blocks", "block 769"))]
    sims = [api.SimScene(ctx, s).upload().init() for s in scs]
    b = api.Batch(ctx, sims).set_tuning(1, 256, 2)
    order, x = [g.storage_order() for g in sims], [s.x for s in scs]
    for _ in range(3):
        b.step(1, dt=[s.dt for s in scs])
        order = [_binned(o, p, s) for o, p, s in zip(order, x, scs)]
        assert all(np.array_equal(g.storage_order(), o) for g, o in zip(sims, order))
        x = [g.check().download()["x"] for g in sims]
    b.close()
    for g in sims:
        g.close()


@gpu
def test_statistics_of_crowded_snow_repeat(ctx):
    """Statistics sum in storage order, so that two runs of a scene agree to the bit."""
    from snow_gb300 import api
    s = _scene(CROWDS["many blocks"], 75)
    runs = []
    for _ in range(3):
        g = api.SimScene(ctx, s, sort_interval=2).upload().init().step(s.dt, 5)
        runs.append(g.stats())
        g.close()
    for r in runs[1:]:
        for k in ("mass", "kinetic_energy", "mean_jp"):
            assert r[k] == runs[0][k]
        assert np.array_equal(r["momentum"], runs[0]["momentum"])
