"""A scene that is set up again starts as a new one does: nothing of the state
before shows (sums not yet consumed, steps the solve may skip)."""
import numpy as np
import pytest

from snow_gb300 import scenes

gpu = pytest.mark.gpu
KEYS = ("x", "v", "FE", "Jp", "volume")


@pytest.fixture(scope="module")
def ctx():
    from snow_gb300 import api
    return api.Context(0)


def _scene(seed, n=3000):
    s = scenes.small_scene(n=n, grid_edge=32, seed=seed, v0=(0.5, -2.0, 0.0))
    s.v += np.random.default_rng(seed).uniform(-0.5, 0.5, s.v.shape).astype(np.float32)
    return s


def _same(a, b):
    return all(np.array_equal(a[k], b[k]) for k in KEYS)


@gpu
@pytest.mark.parametrize("how", ["init twice", "mass and volume kernels", "other state", "fewer particles", "after a grid reset"])
@pytest.mark.parametrize("steps", [0, 5])
def test_set_up_again_is_a_new_scene(ctx, how, steps):
    from snow_gb300 import api, native as N
    s = _scene(621)
    want = api.SimScene(ctx, s).upload().init().step(s.dt, 7).check().download()
    first = _scene(622, 4000 if how == "fewer particles" else s.n)
    g = api.SimScene(ctx, s).upload(first.x, first.v, first.m).init().step(s.dt, steps)
    if how == "after a grid reset":
        g.dispatch(N.K_G_RESET, s.dt)
    g.upload()
    if how == "mass and volume kernels":
        g.dispatch(N.K_G_MASS, s.dt).dispatch(N.K_P_VOLUME, s.dt)
    else:
        g.init()
        if how == "init twice":
            g.init()
    assert _same(g.step(s.dt, 7).check().download(), want)


@gpu
def test_a_solve_after_steps_that_skipped_it(ctx):
    """Snow in free flight skips its solve for up to 240 steps; the state uploaded
    then does not."""
    from snow_gb300 import api
    s = scenes.small_scene(n=3000, grid_edge=32, seed=623, young=1.4e7, v0=(0.0, -1.0, 0.0))
    s.implicit_beta, s.implicit_tolerance, s.implicit_max_iters = 1.0, 1e-5, 30
    v = np.random.default_rng(624).uniform(-2.0, 2.0, s.v.shape).astype(np.float32)
    new = api.SimScene(ctx, s).upload(v=v).init().step(s.dt, 1).solver_report()
    assert new["iterations"] > 0
    g = api.SimScene(ctx, s).upload().init().step(s.dt, 3)
    assert g.solver_report()["iterations"] == 0
    again = g.upload(v=v).init().step(s.dt, 1).solver_report()
    assert again["iterations"] == new["iterations"]


@gpu
@pytest.mark.parametrize("batched", [False, True])
def test_a_condition_of_the_state_before_is_not_reported(ctx, batched):
    from snow_gb300 import api, native as N
    s = _scene(625)
    v = s.v.copy()
    v[3] = np.nan
    g = api.SimScene(ctx, s).upload(v=v).init().step(s.dt, 4)
    with pytest.raises(N.SnowError) as e:
        g.check()
    assert e.value.status == N.SNOW_ENUMERIC
    g.upload().init()
    if batched:
        b = api.Batch(ctx, [g])
        b.step(40, dt=[s.dt])
    else:
        g.step(s.dt, 40)
    want = api.SimScene(ctx, s).upload().init().step(s.dt, 40).check().download()
    assert _same(g.check().download(), want)
