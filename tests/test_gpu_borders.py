"""The FAST step where its tiles meet the grid's border and its work items
their limits, against the FP64 oracle: grids of odd and unequal dimensions
down to one block, snow up to the first and last cells of the grid (the tile
rows of the border blocks lie partly outside it), and item sizes around the
256 particles of a work item. The bound is the single-step parity bound."""
import numpy as np
import pytest

from oracle import oracle as O
from snow_gb300 import scenes

gpu = pytest.mark.gpu
TOL = 1e-5


def _scene(dim, n, seed, lo=None, hi=None):
    """n particles at random in the cells lo .. hi (default: the whole grid)."""
    rng = np.random.default_rng(seed)
    h = 1.0 / 32
    s = scenes.Scene(grid_pos=(0.0, 0.0, 0.0), grid_dim=dim, grid_spacing=h, young=1.4e5, poisson=0.2, hardening=10.0,
                     crit_compression=2.5e-2, crit_stretch=7.5e-3, dt=1e-4)
    lo = np.zeros(3) if lo is None else np.asarray(lo, float)
    hi = np.asarray(dim, float) - 1 if hi is None else np.asarray(hi, float)
    s.x = ((lo + (hi - lo) * rng.uniform(0.001, 0.999, (n, 3))) * h).astype(np.float32)
    s.v = rng.uniform(-2, 2, (n, 3)).astype(np.float32)
    s.m = np.full(n, 400 * h ** 3 / 8, np.float32)
    return s


@gpu
@pytest.mark.parametrize("interval", [1, 8])
@pytest.mark.parametrize("dim,n,lo,hi", [
    ((4, 4, 4), 60, None, None),
    ((5, 9, 33), 700, None, None),
    ((33, 5, 6), 900, None, None),
    ((16, 17, 30), 3000, None, None),
    ((24, 24, 24), 1, (10, 10, 10), (11, 11, 11)),
    ((24, 24, 24), 255, (8, 8, 8), (12, 12, 12)),
    ((24, 24, 24), 256, (8, 8, 8), (12, 12, 12)),
    ((24, 24, 24), 257, (8, 8, 8), (12, 12, 12)),
    ((24, 24, 24), 1025, (0, 0, 20), (4, 4, 23)),
])
def test_border_tiles_and_item_limits_match_the_oracle(dim, n, lo, hi, interval):
    from snow_gb300 import api
    s = _scene(dim, n, 7 + n, lo, hi)
    ctx = api.Context(0)
    g = api.SimScene(ctx, s, sort_interval=interval).upload().init()
    o = O.OracleSim(s, O.EXACT64, vround=False).upload().init()
    g.step(s.dt, 1)
    flip = o.step_with_flip_scale()
    e = O.parity_errors(g.download(), o.state(), flip)["max"]
    assert max(e[k] for k in ("x", "v_flip", "FE", "Jp")) <= TOL, e
    # two more steps (the second binning of interval 1) stay finite and keep the mass
    g.step(s.dt, 2).check()
    st = g.stats()
    assert st["nonfinite"] == 0 and abs(st["mass"] - float(s.m.sum())) <= 1e-5 * float(s.m.sum())
    ctx.close()
