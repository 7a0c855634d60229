"""A call that fails for want of memory leaves the scene as it was, and succeeds once
there is room."""
import numpy as np
import pytest

from snow_gb300 import scenes

gpu = pytest.mark.gpu
KEYS = ("x", "v", "FE", "Jp", "volume")


def _scene():
    return scenes.small_scene(n=6000, grid_edge=32, seed=651, v0=(0.5, -2.0, 0.0))


def _sizes(mode):
    """Bytes a scene holds after its creation, upload and init, and what it steps to."""
    from snow_gb300 import api
    s = _scene()
    ctx = api.Context(0)
    g = api.SimScene(ctx, s, mode=mode)
    created = ctx.bytes_in_use
    uploaded = (g.upload(), ctx.bytes_in_use)[1]
    ready = (g.init(), ctx.bytes_in_use)[1]
    got = g.step(s.dt, 3).check().download()
    ctx.close()
    return created, uploaded, ready, got


def _refused(call):
    from snow_gb300 import native as N
    with pytest.raises(N.SnowError) as e:
        call()
    assert e.value.status == N.SNOW_EBUDGET


@gpu
@pytest.mark.parametrize("mode", ["fast", "reference"])
@pytest.mark.parametrize("fails", ["first array", "half of the arrays", "last array"])
def test_an_upload_without_room_can_be_repeated(mode, fails):
    from snow_gb300 import api, native as N
    mode = N.MODE_FAST if mode == "fast" else N.MODE_REFERENCE
    created, uploaded, ready, want = _sizes(mode)
    s = _scene()
    big = scenes.small_scene(n=200, grid_edge=64, seed=652)  # holds the room until it is closed
    probe = api.Context(0)
    keep = api.SimScene(probe, big)
    held = probe.bytes_in_use
    keep.close(), probe.close()
    assert held > ready - created + 100 * s.n
    room = {"first array": 100, "half of the arrays": (uploaded - created) // 2, "last array": uploaded - created - 1}[fails]
    ctx = api.Context(0, hbm_budget=held + created + room)
    other, g = api.SimScene(ctx, big), api.SimScene(ctx, s, mode=mode)
    for _ in range(2):
        _refused(g.upload)
        assert ctx.bytes_in_use == held + created
    other.close()
    got = g.upload().init().step(s.dt, 3).check().download()
    assert all(np.array_equal(got[k], want[k]) for k in KEYS)
    ctx.close()


@gpu
def test_a_second_upload_without_room_leaves_the_state():
    """Pageable arrays go through a staging buffer; page-locked ones need none."""
    import torch

    from snow_gb300 import api, native as N
    created, uploaded, ready, _ = _sizes(N.MODE_FAST)
    s = _scene()
    assert ready - uploaded > 4 * 7 * s.n  # the first upload's staging buffer
    fe = np.tile(np.eye(3, dtype=np.float32), (s.n, 1, 1)).reshape(-1, 9)
    out = []
    for budget in (0, ready + 100):
        ctx = api.Context(0, hbm_budget=budget)
        g = api.SimScene(ctx, s).upload().init().step(s.dt, 3)
        if budget:
            _refused(lambda: g.upload(FE=fe, FP=fe))
        g.step(s.dt, 3).check()
        x = torch.empty((s.n, 3), dtype=torch.float32, pin_memory=True).numpy()
        assert g.L.snow_scene_download(g.h, N.ptr(x), None, None, None, None, None) == N.SNOW_OK
        out.append(x.copy())
        ctx.close()
    assert np.array_equal(*out)


@gpu
def test_an_init_without_room_can_be_repeated():
    from snow_gb300 import api, native as N
    created, uploaded, ready, want = _sizes(N.MODE_FAST)
    s = _scene()
    big = scenes.small_scene(n=200, grid_edge=64, seed=652)
    probe = api.Context(0)
    keep = api.SimScene(probe, big)
    held = probe.bytes_in_use
    keep.close(), probe.close()
    stage = 4 * 7 * s.n + 1024
    assert ready - uploaded > stage
    ctx = api.Context(0, hbm_budget=held + uploaded + stage)
    other, g = api.SimScene(ctx, big), api.SimScene(ctx, s).upload()
    for _ in range(2):
        _refused(g.init)
    other.close()
    got = g.init().step(s.dt, 3).check().download()
    assert all(np.array_equal(got[k], want[k]) for k in KEYS)
    ctx.close()
