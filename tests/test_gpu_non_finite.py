"""A particle whose stress or momentum is not finite harms its own scene at most
at the nodes of its own stencil: not the particles that share a record with it,
not the items its CTA sums next, not the other scenes of its batch."""
import numpy as np
import pytest

from snow_gb300 import scenes

gpu = pytest.mark.gpu
KEYS = ("x", "v", "FE", "Jp")
STEPS = 6  # before the first look at the counters, which would report the sick scene


@pytest.fixture(scope="module")
def ctx():
    from snow_gb300 import api
    return api.Context(0)


def _healthy(implicit=False):
    scs = [scenes.small_scene(n=n, grid_edge=48, seed=500 + i, v0=(1.0, -3.0, 0.5)) for i, n in enumerate((20_001, 9_999, 7))]
    for s in scs:
        if implicit:
            s.young, s.implicit_beta, s.implicit_tolerance, s.implicit_max_iters = 1.4e7, 1.0, 1e-5, 10
    return scs


def _sick(kind, ctx, implicit=False):
    """A scene set up with what `kind` names, which the calls accept."""
    from snow_gb300 import api
    s = scenes.small_scene(n=30_001, grid_edge=48, seed=510, v0=(0.0, -2.0, 0.0))
    if implicit:
        s.young, s.implicit_beta, s.implicit_max_iters = 1.4e7, 1.0, 10
    fe = np.tile(np.eye(3, dtype=np.float32), (s.n, 1, 1))
    fp = fe.copy()
    if kind == "poisson":
        s.poisson = 0.5  # lambda is infinite, times J - 1 = 0
    elif kind == "young":
        s.young = np.inf
    elif kind == "FE":
        fe[::50, 1, 2] = np.nan
    elif kind == "FP":
        fp[::50, 0, 0] = np.nan
    return api.SimScene(ctx, s).upload(FE=fe.reshape(-1, 9), FP=fp.reshape(-1, 9)).init()


@gpu
@pytest.mark.parametrize("kind", ["poisson", "young", "FE", "FP"])
@pytest.mark.parametrize("sick_implicit", [False, True])
def test_a_sick_scene_leaves_the_others_of_its_batch_alone(ctx, kind, sick_implicit):
    from snow_gb300 import api
    scs = _healthy()
    alone = [api.SimScene(ctx, s).upload().init().step(s.dt, STEPS).download() for s in scs]
    sims = [api.SimScene(ctx, s).upload().init() for s in scs]
    sims.insert(1, _sick(kind, ctx, sick_implicit))
    api.Batch(ctx, sims).step(STEPS, dt=[scs[0].dt] * len(sims))
    del sims[1]
    for a, g in zip(alone, sims):
        got = g.download()
        assert all(np.array_equal(a[k], got[k]) for k in KEYS)


@gpu
@pytest.mark.parametrize("kind", ["poisson", "FE", "FP"])
def test_a_sick_solve_leaves_the_others_of_its_batch_alone(ctx, kind):
    """Semi-implicit scenes: their float sums of K u have no fixed order, so that two
    runs differ by what the solve leaves open, 1e-5 of the velocity (here up to
    4 m/s) a step: 2 x 6 x 4e-5 m/s, and 1e-4 s of that a step in position."""
    from snow_gb300 import api
    scs = _healthy(implicit=True)
    alone = [api.SimScene(ctx, s).upload().init().step(s.dt, STEPS).download() for s in scs]
    sims = [api.SimScene(ctx, s).upload().init() for s in scs]
    sims.insert(1, _sick(kind, ctx, implicit=True))
    api.Batch(ctx, sims).step(STEPS, dt=[scs[0].dt] * len(sims))
    del sims[1]
    for s, a, g in zip(scs, alone, sims):
        got = g.download()
        assert np.abs(got["v"] - a["v"]).max() <= 1e-3
        assert np.abs(got["x"] - a["x"]).max() <= 1e-3 * s.dt * STEPS + 1e-6


@gpu
@pytest.mark.parametrize("where", ["FE", "v"])
def test_set_up_sums_outside_a_sick_particles_stencil(ctx, where):
    """The P2G of an uploaded state with NaN in 40 particles of one corner: the sums
    of all nodes beyond their 4 x 4 x 4 stencils are those of the same state without
    them."""
    from snow_gb300 import api, native as N
    s = scenes.small_scene(n=20_001, grid_edge=48, seed=520, v0=(0.5, -2.0, 0.25))
    sick = np.argsort(s.x.sum(1))[:40]
    fe = np.tile(1.001 * np.eye(3, dtype=np.float32), (s.n, 1, 1))
    fe[sick] = np.eye(3)  # no stress: the scale is the others'
    grids = []
    for nan in (False, True):
        f, v = fe.copy(), s.v.copy()
        if nan:
            (f if where == "FE" else v).reshape(s.n, -1)[sick, 1] = np.nan
        g = api.SimScene(ctx, s).upload(v=v, FE=f.reshape(-1, 9)).init()
        g.dispatch(N.K_P2G, s.dt)
        grids.append(g.grid())
        g.close()
    beyond = np.ones(s.grid_dim[::-1], bool)
    for cell in ((s.x[sick] - np.asarray(s.grid_pos)) / s.grid_spacing).astype(int):
        beyond[tuple(slice(c - 1, c + 3) for c in cell[::-1])] = False
    beyond = beyond.reshape(-1)
    for k in ("mass", "mom", "force"):
        assert np.count_nonzero(grids[0][k][beyond]) > 1000
        assert np.array_equal(grids[1][k][beyond], grids[0][k][beyond]), k
        assert np.all(np.isfinite(grids[1][k])), k
