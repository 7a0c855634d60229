"""A job whose particles turn non-finite fails alone: the jobs that share its batch
finish with the state they have alone."""
import numpy as np
import pytest

from snow_gb300 import scenes

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("chunk", [5, 16, 64])
def test_a_sick_job_fails_alone(chunk):
    from snow_gb300 import api, native as N
    jobs = [scenes.small_scene(n=n, grid_edge=32, seed=670 + i, v0=(0.5, -1.0, 0.0)) for i, n in enumerate((3001, 2000, 999, 4000))]
    steps = [130, 90, 100, 70]
    sick = jobs[1]
    sick.v = sick.v.copy()
    sick.v[7] = np.nan
    srv = api.Server(0, chunk_steps=chunk)
    try:
        ids = [srv.submit(s, steps=k, keep_state=True) for s, k in zip(jobs, steps)]
        srv.drain(120.0)
        res = {r["id"]: r for r in srv.poll()}
        ctx = api.Context(0)
        for jid, s, k in zip(ids, jobs, steps):
            if s is sick:
                assert res[jid]["status"] == N.SNOW_ENUMERIC
                continue
            assert res[jid]["status"] == N.SNOW_OK
            want = api.SimScene(ctx, s).upload().init().step(s.dt, k).check().download()
            got = srv.fetch(jid, s.n)
            assert all(np.array_equal(want[q], got[q]) for q in ("x", "v", "FE", "Jp"))
        st = srv.stats()
        assert st["completed"] == 3 and st["failed"] == 1
        ctx.close()
    finally:
        srv.close()
