"""Single dispatches leave the state that a step relies on as it is."""
import numpy as np
import pytest

from snow_gb300 import scenes

gpu = pytest.mark.gpu
KEYS = ("x", "v", "FE", "Jp")


@pytest.fixture(scope="module")
def ctx():
    from snow_gb300 import api
    return api.Context(0)


@gpu
@pytest.mark.parametrize("times", [1, 2, 5])
@pytest.mark.parametrize("before", [0, 3, 40])
def test_a_rigid_advance_between_steps_moves_the_colliders_alone(ctx, before, times):
    """With static walls it moves nothing: the steps after it are those without it."""
    from snow_gb300 import api, native as N
    s = scenes.small_scene(n=3000, grid_edge=32, seed=611, v0=(0.5, -2.0, 0.0))
    runs = []
    for advance in (0, times):
        g = api.SimScene(ctx, s).upload().init().step(s.dt, before)
        for _ in range(advance):
            g.dispatch(N.K_RIGID_ADVANCE, s.dt)
        runs.append(g.step(s.dt, 20).check().download())
        g.close()
    assert all(np.array_equal(runs[0][k], runs[1][k]) for k in KEYS)
    assert np.abs(runs[0]["v"][:, 1]).max() > 2.0  # falling


@gpu
def test_a_rigid_advance_moves_what_a_step_would(ctx):
    from snow_gb300 import api, native as N
    s = scenes.small_scene(n=500, grid_edge=16, seed=612)
    s.colliders += [scenes.Collider(pos=(0.5, 0.05 + 0.01 * i, 0.5), type=1, radius=0.01, vel=(0.0, 0.5, -0.1 * i)) for i in range(40)]
    a, b = (api.SimScene(ctx, s).upload().init() for _ in range(2))
    a.dispatch(N.K_RIGID_ADVANCE, 1e-3)
    b.step(1e-3, 1)
    assert np.array_equal(a.colliders(), b.colliders())
    assert np.abs(a.colliders()[-1] - np.array([0.5, 0.4405, 0.5 - 3.9e-3])).max() < 1e-6
