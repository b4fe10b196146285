"""Calls from several host threads at once, buffers and a stream each."""
import threading

import numpy as np
import pytest
import torch

from dsplat import _native as N
from gpu_util import F, T

pytestmark = pytest.mark.gpu


def test_tile_lists_of_different_views_at_once(dev):
    """400 and 256 superblocks: the superblock scatter needs 53 KB and 50 KB
    of shared memory, both above what a kernel gets without asking, and
    neither call may lower the limit under the other."""
    L = N.lib()
    rng = np.random.default_rng(0)
    n, cap = 200, 1 << 16
    xyd = T(rng.uniform(0, 1, (n, 3)).astype(np.float32) * [900, 900, 1], dev, torch.float32)
    aabb = torch.cat([xyd[:, :2] - 5, xyd[:, :2] + 5], 1).contiguous()
    calls, outs = [], []
    for side in (1280, 1024):
        tiles = side // 8
        ws = torch.empty(L.dsplat_tile2idx_workspace_size(n, tiles, tiles, cap), dtype=torch.uint8, device=dev)
        t2i = torch.empty(tiles * tiles + 1, dtype=torch.int32, device=dev)
        i2p = torch.zeros(cap, dtype=torch.int32, device=dev)
        stream = torch.cuda.Stream(dev)
        args = (stream.cuda_stream, n, xyd.data_ptr(), aabb.data_ptr(), side, side, 8, t2i.data_ptr(), i2p.data_ptr(),
                cap, None, ws.data_ptr(), ws.numel())
        calls.append((stream, args))
        outs.append((t2i, i2p, ws))
    torch.cuda.synchronize(dev)
    want = []
    for (stream, args), (t2i, i2p, _) in zip(calls, outs):
        N.check(L.dsplat_gauss_tile2idx_idx2pnt(*args), "lists")
        stream.synchronize()
        want.append((F(t2i).copy(), F(i2p).copy()))
    refused = [0, 0]

    def work(k):
        stream, args = calls[k]
        for i in range(20000):
            refused[k] += L.dsplat_gauss_tile2idx_idx2pnt(*args) != 0
            if i % 100 == 99:
                stream.synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize(dev)
    assert refused == [0, 0]
    for (t2i, i2p, _), (a, b) in zip(outs, want):
        assert np.array_equal(F(t2i), a) and np.array_equal(F(i2p), b)
