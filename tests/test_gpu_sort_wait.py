"""The static sort's blocks wait for one another for a bounded time: a wait that
runs out is reported, and the sort stays usable."""
import ctypes as C

import numpy as np
import pytest

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("n", [1, 100003, 262144])
def test_a_wait_that_runs_out_is_reported_once(n):
    import torch

    from snow_gb300 import native as N
    L = N.load()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    k = np.random.default_rng(n).integers(0, 1 << 20, size=n, dtype=np.uint32)
    keys = torch.from_numpy(k.view(np.int32).copy()).cuda()
    out, perm = torch.empty_like(keys), torch.empty_like(keys)
    args = (keys.data_ptr(), out.data_ptr(), perm.data_ptr(), n, 20, stream)
    assert L.snow_sort_static_check(stream) == N.SNOW_OK
    # one arrival more than there are blocks: nothing makes it, and each block gives up after 1 ms
    assert L.snow_sort_keys_static_limited(*args, 1_000_000, 1) == N.SNOW_OK
    assert L.snow_sort_keys_static(*args) == N.SNOW_OK  # a sort that ends well does not hide it
    assert L.snow_sort_static_check(stream) == N.SNOW_ETIMEDOUT
    assert L.snow_sort_static_check(stream) == N.SNOW_OK
    want = np.argsort(k, kind="stable").astype(np.uint32)
    assert np.array_equal(perm.cpu().numpy().view(np.uint32), want)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), k[want])
