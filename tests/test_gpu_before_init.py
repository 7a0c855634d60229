"""Calls that need no set-up work on a scene that has none: the device's copy of the
scene's description is there whenever a kernel reads it. Steps are refused."""
import numpy as np
import pytest

from oracle import oracle as O
from snow_gb300 import scenes

gpu = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from snow_gb300 import api
    return api.Context(0)


def _uploaded(g, s):
    got = g.download()
    assert np.array_equal(got["x"], s.x) and np.array_equal(got["v"], s.v)
    assert np.array_equal(got["FE"], np.tile(np.eye(3, dtype=np.float32), (s.n, 1, 1)))
    assert np.all(got["Jp"] == 1.0) and np.all(got["volume"] == 0.0)


@gpu
@pytest.mark.parametrize("capacity", [0, 5000])
def test_an_uploaded_scene_can_be_read(ctx, capacity):
    from snow_gb300 import api
    s = scenes.small_scene(n=3001, grid_edge=32, seed=641, v0=(1.0, -2.0, 0.5))
    g = api.SimScene(ctx, s, capacity=capacity).upload()
    _uploaded(g, s)
    st = g.stats()
    assert st["n"] == s.n and st["nonfinite"] == 0
    assert abs(st["mass"] - s.m.astype(np.float64).sum()) <= 1e-6 * s.m.sum()
    keys, perm = g.cell_keys()
    _, want, want_perm = O.cell_keys(s.x, s.grid_pos, s.grid_dim, s.grid_spacing)
    assert np.array_equal(keys, want) and np.array_equal(perm, want_perm)
    assert not np.any(g.grid()["mass"])
    # another upload, of fewer particles, before and after a set-up
    t = scenes.small_scene(n=1500, grid_edge=32, seed=642)
    for _ in range(2):
        g.upload(t.x, t.v, t.m)
        _uploaded(g, t)
        assert np.array_equal(g.cell_keys()[0], O.cell_keys(t.x, t.grid_pos, t.grid_dim, t.grid_spacing)[1])
        g.upload().init().step(s.dt, 2).check()
    g.close()


@gpu
@pytest.mark.parametrize("dt", [1e-3, 5e-4])
def test_colliders_of_an_uploaded_scene_can_be_advanced(ctx, dt):
    from snow_gb300 import api, native as N
    s = scenes.small_scene(n=100, grid_edge=16, seed=643)
    s.colliders.append(scenes.Collider(pos=(0.5, 0.1, 0.5), type=1, radius=0.05, vel=(0.0, 1.0, 0.0)))
    g = api.SimScene(ctx, s).upload()
    g.dispatch(N.K_RIGID_ADVANCE, dt)
    assert abs(g.colliders()[-1][1] - (0.1 + dt)) < 1e-7
    g.close()


@gpu
def test_a_batch_does_not_step_a_scene_that_is_not_set_up(ctx):
    from snow_gb300 import api, native as N
    scs = [scenes.small_scene(n=900, grid_edge=16, seed=644 + i) for i in range(2)]
    sims = [api.SimScene(ctx, s).upload().init() for s in scs]
    b = api.Batch(ctx, sims)
    dts = [s.dt for s in scs]
    b.step(2, dt=dts)
    sims[1].upload()
    with pytest.raises(N.SnowError) as e:
        b.step(1, dt=dts)
    assert e.value.status == N.SNOW_ESTATE
    sims[1].init()
    b.step(2, dt=dts)
    want = api.SimScene(ctx, scs[1]).upload().init().step(dts[1], 2).download()
    got = sims[1].check().download()
    assert all(np.array_equal(want[k], got[k]) for k in ("x", "v", "FE", "Jp"))
    b.close()
