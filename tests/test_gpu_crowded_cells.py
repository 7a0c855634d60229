"""Cells of more than 32 of an item's particles are summed in shares of up to 16 by
several half-warps: at the sizes where shares begin and end, against items cut
otherwise (equal bits: the sums are integers) and against the FP64 oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from snow_gb300 import scenes

gpu = pytest.mark.gpu
KEYS = ("x", "v", "FE", "Jp")

# particles of the cells 0, 1, ... of blocks in a row
LAYOUTS = {
    "32 and 33": [[32] * 8, [33] * 7, [31, 33, 32, 1, 34]],
    "odd starts": [[1, 33, 1, 47, 48, 49, 3], [7, 65, 5, 64, 0, 0, 63]],
    "whole items": [[256], [255, 1], [257], [0, 0, 256, 256, 40]],
    "many items": [[300, 700, 20, 1500], [5000]],
    "beside ordinary ones": [[8] * 20 + [40] + [8] * 20 + [200] + [8] * 8],
}


def _scene(layout, seed, **kw):
    rng = np.random.default_rng(seed)
    s = scenes.unit_box_scene(32, young=1.4e5, poisson=0.2, hardening=10.0, crit_compression=2.5e-2,
                              crit_stretch=7.5e-3, dt=1e-4, name="crowd", **kw)
    at = [(8 + 4 * b + (c & 3), 12 + (c >> 2 & 3), 12 + (c >> 4))
          for b, cells in enumerate(LAYOUTS[layout]) for c, n in enumerate(cells) for _ in range(n)]
    s.x = ((np.array(at) + rng.uniform(0.02, 0.98, (len(at), 3))) * s.grid_spacing).astype(np.float32)
    s.v = rng.uniform(-0.5, 0.5, s.x.shape).astype(np.float32) + np.float32([0.3, -1.0, 0.2])
    s.m = np.full(len(at), scenes.SNOW_DENSITY * s.grid_spacing ** 3 / 64.0, np.float32)
    return s


@pytest.fixture(scope="module")
def ctx():
    from snow_gb300 import api
    return api.Context(0)


@gpu
@pytest.mark.parametrize("layout", list(LAYOUTS))
def test_crowded_cells_sum_alike_however_items_are_cut(ctx, layout):
    from snow_gb300 import api
    s = _scene(layout, 661)
    runs = []
    for items, ctas in ((256, 2), (256, 1), (144, 2), (96, 2), (64, 1)):
        g = api.SimScene(ctx, s)
        g.set_tuning(4, items, ctas)
        runs.append(g.upload().init().step(s.dt, 9).check().download())
        g.close()
    for r in runs[1:]:
        assert all(np.array_equal(r[k], runs[0][k]) for k in KEYS)


@gpu
@pytest.mark.parametrize("layout", list(LAYOUTS))
def test_a_step_of_crowded_cells_matches_the_oracle(ctx, layout):
    from snow_gb300 import api
    s = _scene(layout, 662)
    g = api.SimScene(ctx, s).upload().init().step(s.dt, 1).check()
    o = O.OracleSim(s, mode=O.EXACT64).upload().init()
    flip = o.step_with_flip_scale()
    e = O.parity_errors(g.download(), o.state(), flip)
    g.close()
    assert max(e["max"][k] for k in ("x", "v_flip", "FE", "Jp")) <= 1e-5


@gpu
@pytest.mark.parametrize("layout", list(LAYOUTS))
def test_a_solve_of_crowded_cells_matches_the_oracle(ctx, layout):
    """The solve's K u (float sums): no further from the exact solve than its input,
    v*, is from the exact one, and the solve's tolerance of 1e-6 five times."""
    from snow_gb300 import api, native as N
    speeds = []
    for beta in (0.0, 1.0):
        s = _scene(layout, 663)
        s.young, s.dt = 1.4e7, 5e-3
        s.implicit_beta, s.implicit_tolerance, s.implicit_max_iters = beta, 1e-6, 100
        g = api.SimScene(ctx, s).upload().init()
        g.dispatch(N.K_P2G, s.dt)
        g.dispatch(N.K_G_FORCE, s.dt)
        speeds.append(g.grid()["vstar"].astype(np.float64))
        g.close()
    o = O.OracleSim(s, O.EXACT64, vround=False).upload().init()
    for phase in (O.PH_RESET, O.PH_P2G):
        o.phase(phase)
    o.phase(O.PH_GRID, s.dt)
    vstar, m = o.grid()["vstar"].copy(), o.grid()["mass"][:, None]
    o.set_implicit(1.0, 1e-10, 200)
    o.phase(O.PH_IMPLICIT, s.dt)
    norm = lambda a: float(np.sqrt(np.sum(m * a * a)))
    err_in, err_out = norm(speeds[0] - vstar) / norm(vstar), norm(speeds[1] - o.grid()["vstar"]) / norm(vstar)
    assert err_in <= 1e-3
    assert err_out <= max(err_in, 1e-6) + 5e-6
