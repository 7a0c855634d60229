"""snow_sort_keys_static where its tiles of 2,048 keys and passes of 8 bits
end: one key to the largest number, every number of passes, keys that are all
alike, in place and captured in a CUDA graph, against numpy's stable argsort
(whole numbers: equal)."""
import ctypes as C

import numpy as np
import pytest

gpu = pytest.mark.gpu


def _call(keys, out, perm, n, bits, stream):
    from snow_gb300 import native as N
    st = N.load().snow_sort_keys_static(keys.data_ptr(), out.data_ptr(), perm.data_ptr(), n, bits, C.c_void_p(stream))
    assert st == N.SNOW_OK


@gpu
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("n,bits,distinct", [(1, 1, 1), (31, 8, 5), (2047, 9, 300), (2048, 16, 2048), (2049, 17, 9),
                                             (6145, 24, 6000), (100003, 25, 50000), (262143, 32, 1 << 20), (262144, 32, 1),
                                             (262144, 7, 128)])
def test_sort_sizes_and_passes(n, bits, distinct, in_place):
    import torch
    rng = np.random.default_rng(n + bits)
    top = 1 << bits
    pool = rng.integers(0, top, size=distinct, dtype=np.uint64)
    k = pool[rng.integers(0, distinct, size=n)].astype(np.uint32)
    want = np.argsort(k, kind="stable").astype(np.uint32)
    keys = torch.from_numpy(k.view(np.int32).copy()).cuda()
    out = keys if in_place else torch.empty_like(keys)
    perm = torch.full_like(keys, -1)
    _call(keys, out, perm, n, bits, torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(perm.cpu().numpy().view(np.uint32), want)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), k[want])


@gpu
def test_sort_in_a_captured_graph():
    import torch
    n = 50001
    rng = np.random.default_rng(3)
    k = rng.integers(0, 1 << 20, size=n, dtype=np.uint32)
    keys = torch.from_numpy(k.view(np.int32).copy()).cuda()
    out, perm = torch.empty_like(keys), torch.empty_like(keys)
    _call(keys, out, perm, n, 20, torch.cuda.current_stream().cuda_stream)  # looks the scratch up
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        _call(keys, out, perm, n, 20, torch.cuda.current_stream().cuda_stream)
    k2 = rng.integers(0, 1 << 20, size=n, dtype=np.uint32)
    for data in (k, k2):
        keys.copy_(torch.from_numpy(data.view(np.int32)))
        out.zero_(), perm.zero_()
        g.replay()
        torch.cuda.synchronize()
        want = np.argsort(data, kind="stable").astype(np.uint32)
        assert np.array_equal(perm.cpu().numpy().view(np.uint32), want)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), data[want])
