"""REFERENCE mode where its blocks of 64 particles and groups of eight lanes
end: particle counts around them, against the oracle's FP32 restatement of the
shaders. The integer sums of a step have the same value however the pairs are
dealt out, so that two runs and two orders of the particles give equal bits."""
import numpy as np
import pytest

from oracle import oracle as O
from snow_gb300 import scenes

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("n", [1, 7, 63, 64, 65, 257, 4099])
def test_reference_steps_at_block_edges(n):
    from snow_gb300 import api, native as N
    ctx = api.Context(0)
    s = scenes.small_scene(n=n, grid_edge=24, seed=5 + n, v0=(0.5, -2.0, 0.25))
    bufs = s.std140()
    r = api.SimScene(ctx, s, mode=N.MODE_REFERENCE).upload_std140(*bufs).init().step(s.dt, 2)
    q = O.OracleSim(s, mode=O.FAITHFUL32).upload_std140(*bufs).init().step(n=2)
    got, want = r.download_std140(), q.state_std140()
    assert np.abs(got[0] - want[0]).max() <= 1e-6
    assert np.abs(got[1][:, :3].astype(np.int64) - want[1][:, :3]).max() <= 10000
    perm = np.random.default_rng(n).permutation(n)
    t = api.SimScene(ctx, s, mode=N.MODE_REFERENCE).upload_std140(*(b[perm] for b in bufs)).init().step(s.dt, 2)
    for a, b in zip(got, t.download_std140()):
        assert np.array_equal(a[perm], b)
    ctx.close()
