"""A set-up starts the re-binning schedule anew: what was learned of the state before
(speeds, particles outside their tiles) is not that of the new one. Read from the
order in which the particles lie, which a binning changes once they have moved."""
import numpy as np
import pytest

from snow_gb300 import scenes

gpu = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from snow_gb300 import api
    return api.Context(0)


def _scene(seed, speed):
    s = scenes.small_scene(n=6000, grid_edge=64, seed=seed, v0=(speed, 0.0, 0.0), center=(0.3, 0.5, 0.5))
    s.dt, s.gravity, s.young = 1e-3, (0.0, 0.0, 0.0), 1.0
    return s


FAST, SLOW = 6.7, 0.1  # 0.43 of a cell a step (3.4 in eight: another order) and 1/156


def _steps_to_binning(g, step, most):
    order = g.storage_order()
    for k in range(1, most + 1):
        step()
        if not np.array_equal(g.storage_order(), order):
            return k
    return most + 1


@gpu
@pytest.mark.parametrize("others", [0, 2])
def test_a_batch_after_an_upload_of_faster_snow(ctx, others):
    """A slow batch re-bins every 32 steps; with fast snow, every eight unless particles
    are seen to leave their tiles: the ninth step is the first to bin."""
    from snow_gb300 import api
    slow, fast = _scene(631, SLOW), _scene(632, FAST)
    sims = [api.SimScene(ctx, slow).upload().init() for _ in range(1 + others)]
    b = api.Batch(ctx, sims)
    dts = [slow.dt] * len(sims)
    b.step(17, dt=dts)  # a look at the counters, and a step
    g = sims[0]
    g.upload(fast.x, fast.v, fast.m).init()
    assert _steps_to_binning(g, lambda: b.step(1, dt=dts), 20) <= 9
    for g in sims:
        g.check()
    b.close()


@gpu
def test_a_scene_with_a_chosen_interval_after_an_upload_of_slower_snow(ctx):
    """Fast snow brings the interval down from the chosen one, slow snow starts at it:
    64 steps take 7 binnings (after 8, 16, .. 56)."""
    from snow_gb300 import api
    slow, fast = _scene(633, SLOW), _scene(634, FAST)
    g = api.SimScene(ctx, fast, sort_interval=8).upload().init().step(fast.dt, 30)
    assert g.phase_times(reset=True)["binnings"] > 10
    g.upload(slow.x, slow.v, slow.m).init().step(slow.dt, 64).check()
    assert g.phase_times()["binnings"] == 7


@gpu
def test_the_interval_stays_within_what_the_speeds_allow(ctx):
    """Snow in free flight at a twentieth of a cell a step may go 0.8 / 0.05 = 16 steps
    between binnings, however long all goes well."""
    from snow_gb300 import api
    s = _scene(635, 0.05 * 15.625)  # 0.05 of h = 1/64 m in 1 ms
    g = api.SimScene(ctx, s).upload().init()
    binned = [0]
    for k in range(256):
        before = g.phase_times()["binnings"]
        if g.step(s.dt, 1).phase_times()["binnings"] > before:
            binned.append(k)
    assert len(binned) > 10 and np.diff(binned).max() <= 16
    g.check()
    g.close()


@gpu
@pytest.mark.parametrize("beyond", [0.3, 3.0])
def test_particles_outside_the_grid_are_no_reason_to_bin(ctx, beyond):
    """A third of the particles lie beyond the grid's end, in no tile wherever they are
    binned to: slow snow still takes 32 steps between binnings (after the first eight)."""
    from snow_gb300 import api
    s = _scene(636, SLOW)
    s.colliders = []
    s.x[::3, 0] += np.float32(0.7 + beyond)
    g = api.SimScene(ctx, s).upload().init().step(s.dt, 128).check()
    assert g.phase_times()["binnings"] <= 128 // 32
    g.close()


@gpu
def test_an_interval_shortened_once_is_not_shortened_twice(ctx):
    """A snowball that falls at 0.30 to 0.33 of a cell a step, hits the ground and
    slides: two to three steps between binnings while it falls. That particles left
    their tiles is counted in one more look after the interval was shortened for it,
    which is no reason to bin every step for the next hundred."""
    from snow_gb300 import api
    s = scenes.small_scene(n=60_000, grid_edge=64, seed=3, v0=(2.0, -4.0, 1.0), young=2e4)
    s.dt = 1e-3
    g = api.SimScene(ctx, s).upload().init().step(s.dt, 72)
    g.phase_times(reset=True)
    assert g.step(s.dt, 64).phase_times(reset=True)["binnings"] <= 32
    g.step(s.dt, 64).phase_times(reset=True)
    assert g.step(s.dt, 64).check().phase_times()["binnings"] <= 16  # 0.08 of a cell: seven
    g.close()
