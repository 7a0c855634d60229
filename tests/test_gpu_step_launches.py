"""How the FAST step is launched does not show in its results: scenes are the
same bit for bit alone and in a batch of any size (the step's start and its
prefixes are formed by warps over 8 and 32 scenes)."""
import numpy as np
import pytest

from snow_gb300 import scenes

gpu = pytest.mark.gpu
KEYS = ("x", "v", "FE", "Jp")


def _same(a, b):
    return all(np.array_equal(a[k], b[k]) for k in KEYS)


@gpu
@pytest.mark.parametrize("count", [1, 8, 9, 32, 33, 70])
def test_batches_of_any_number_of_scenes_match_each_alone(count):
    from snow_gb300 import api
    kinds = [scenes.small_scene(n=200 + 37 * i, grid_edge=(17, 24, 9)[i % 3], seed=300 + i, v0=(0.5, -1.0 - i, 0.0))
             for i in range(5)]
    ctx = api.Context(0)
    alone = [api.SimScene(ctx, s).upload().init().step(s.dt, 11).download() for s in kinds]
    scs = [kinds[i % 5] for i in range(count)]
    sims = [api.SimScene(ctx, s).upload().init() for s in scs]
    api.Batch(ctx, sims).step(11, dt=[s.dt for s in scs])
    for i, g in enumerate(sims):
        assert _same(g.check().download(), alone[i % 5]), i
    ctx.close()


@gpu
@pytest.mark.parametrize("interval", [0, 1, 3, 6, 32])
def test_steps_in_one_call_or_in_many_are_the_same(interval):
    """One call of 75 steps (graphs of several steps from its first on), calls of
    one step, mixed calls (a graph of several steps from some point on), and
    plain launches."""
    from snow_gb300 import api
    s = scenes.small_scene(n=2500, grid_edge=32, seed=41, v0=(1.0, -3.0, 0.5))
    ctx = api.Context(0)
    runs = []
    for calls, graphs in (([75], True), ([1] * 75, True), ([5, 7, 4, 4, 4, 4, 4, 4, 4, 20, 15], True), ([75], False),
                          ([40, 35], False)):
        assert sum(calls) == 75
        ctx.set_graphs(graphs)
        g = api.SimScene(ctx, s, sort_interval=interval).upload().init()
        for n in calls:
            g.step(s.dt, n)
        runs.append(g.check().download())
        g.step(0.5 * s.dt, 40)  # another time step: other graphs
        runs[-1]["then"] = g.check().download()
        g.close()
    ctx.set_graphs(True)
    for r in runs[1:]:
        assert _same(r, runs[0]) and _same(r["then"], runs[0]["then"])
    ctx.close()


@gpu
@pytest.mark.parametrize("interval", [0, 1])
@pytest.mark.parametrize("n", [1, 2500, (1 << 20) - 1, 1 << 20, (1 << 20) + 1])
def test_chained_launches_match_separate_ones(n, interval):
    """A profiled step waits for each of its kernels' groups; the others' kernels
    are chained up to 2^20 particles."""
    from snow_gb300 import api
    s = scenes.small_scene(n=n, grid_edge=128 if n > 10000 else 32, seed=43, v0=(1.0, -3.0, 0.5))
    ctx = api.Context(0)
    runs = []
    for profiled, graphs in ((True, True), (False, True), (False, False)):
        ctx.set_profiling(profiled)
        ctx.set_graphs(graphs)
        g = api.SimScene(ctx, s, sort_interval=interval).upload().init().step(s.dt, 41)
        runs.append(g.check().download())
        g.close()
    for r in runs[1:]:
        assert _same(r, runs[0])
    ctx.close()


@gpu
@pytest.mark.parametrize("n", [40, 4096, 33000, 70000, 3 * 304 * 256, 3 * 304 * 256 + 1])
def test_fitted_items_give_the_results_of_full_ones(n):
    """Items sized by the binning (up to three rounds of the GPU's CTAs) against
    items of up to 256: alone, in a batch that the scenes enter after their set-up,
    and alone again."""
    from snow_gb300 import api
    edge = 32 if n < 10000 else 64 if n < 100000 else 96
    s = scenes.small_scene(n=n, grid_edge=edge, seed=47, v0=(1.0, -3.0, 0.5))
    t = scenes.small_scene(n=900, grid_edge=24, seed=48)
    ctx = api.Context(0)
    out = []
    for full in (True, False):
        sims = [api.SimScene(ctx, c) for c in (s, t)]
        if full:
            for g in sims:
                g.set_tuning(8, 256, 2)
        for g in sims:
            g.upload().init().step(s.dt, 10)
        got = [g.check().download() for g in sims]
        b = api.Batch(ctx, sims)
        b.step(13, dt=[s.dt, t.dt])
        got += [g.check().download() for g in sims]
        b.close()
        got += [g.step(s.dt, 20).check().download() for g in sims]
        out.append(got)
    for a, b in zip(*out):
        assert _same(a, b)
    ctx.close()


@gpu
@pytest.mark.parametrize("kind,n", [("dense", 200_003), ("dense", 70_001), ("sphere", 300_000), ("sphere", 9000)])
def test_the_work_split_does_not_show_in_the_results(kind, n):
    """Units of whole runs, of two items and of single ones: item sizes and CTAs
    that take the items through three, five and more rounds of the CTAs; dense
    snow has runs of hundreds of items, an odd number among them."""
    from snow_gb300 import api
    s = scenes.small_scene(n=n, grid_edge=32 if kind == "dense" else 96, seed=51, v0=(0.5, -2.0, 0.0))
    if kind == "dense":  # five blocks, 16,000 to 64,000 particles each (at 200k), masses to match
        rng = np.random.default_rng(52)
        cells = np.array([[8, 8, 8], [12, 8, 8], [16, 8, 8], [8, 16, 12], [20, 20, 20]])[rng.choice(
            5, n, p=[0.1, 0.1, 0.2, 0.28, 0.32])]
        s.x = ((cells + rng.uniform(0.6, 3.4, (n, 3))) * s.grid_spacing).astype(np.float32) + np.float32(s.grid_pos[0])
        s.m = (s.m / 100).astype(np.float32)
    ctx = api.Context(0)
    first = None
    for items, ctas in ((256, 2), (256, 1), (128, 2), (64, 2), (64, 1)):
        g = api.SimScene(ctx, s)
        g.set_tuning(4, items, ctas)
        out = g.upload().init().step(s.dt, 9).check().download()
        g.close()
        first = first or out
        assert _same(out, first), (items, ctas)
    ctx.close()


@gpu
@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("n,speed,young", [(3000, 0.01, 1.4e5), (3000, 2.0, 1.4e5), (20_001, 5.0, 1.4e5),
                                           (20_001, 20.0, 1.4e7), (60_000, 3.0, 1e3)])
def test_first_steps_with_forces_that_outgrow_the_scale(n, speed, young, graphs):
    """Snow at rest in itself that is given random velocities: its first step's
    forces are orders of magnitude above the scale chosen from a state without
    any. A scene's own first step sums such particles in shared memory, a batch's by
    atomics on the grid: the same integers."""
    from snow_gb300 import api
    s = scenes.small_scene(n=n, grid_edge=32 if n < 10000 else 64, seed=61, young=young, dt=2e-5)
    s.v = np.random.default_rng(62).uniform(-speed, speed, (n, 3)).astype(np.float32)
    s.v[: n // 3] *= 1e-3  # and some that stay in range, in the same warps' neighbourhoods
    ctx = api.Context(0)
    ctx.set_graphs(graphs)
    alone = api.SimScene(ctx, s).upload().init()
    other = api.SimScene(ctx, s).upload().init()
    batch = api.Batch(ctx, [other])
    wide = []
    for steps in (1, 1, 6):
        alone.step(s.dt, steps)
        batch.step(steps, dt=[s.dt])
        assert _same(alone.check().download(), other.check().download())
        wide.append((alone.phase_times()["wide"], other.phase_times()["wide"]))
    assert all(a == b for a, b in wide)
    assert wide[0][0] > n // 2 or speed < 1
    ctx.close()
