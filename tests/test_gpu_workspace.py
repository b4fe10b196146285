"""A batch's workspace in memory that an earlier batch of the same layout used."""
import numpy as np
import pytest
import torch

from dsplat import scenes
from dsplat.gauss import GaussBatch
from gpu_util import F, params_of

pytestmark = pytest.mark.gpu


def test_memory_of_an_earlier_batch(dev):
    """The earlier batch left the mark of a clean gradient buffer behind its
    end; other tensors have written over the buffer since."""
    sc = scenes.config0(seed=1, n=30000, size=(160, 120))
    p = params_of(sc, dev)
    up = torch.rand(160 * 120 * 3, device=dev)

    def gradients(batch):
        batch.forward(p)
        grads = {k: torch.zeros_like(v) for k, v in p.items()}
        batch.backward(p, grads, up)
        return {k: F(v).astype(np.float64) for k, v in grads.items()}

    batch = GaussBatch(sc.n, sc.cameras, 16, -1, pair_capacity=1 << 20, device=dev)
    total, used = int(batch.layout.total_bytes), int(batch.layout.off_grad2d) + 48 * sc.n
    want = gradients(batch)
    memory = batch.ws
    del batch
    memory[:used].fill_(0x3f)  # 0x3f3f3f3f: 0.747
    torch.cuda.synchronize(dev)
    empty = torch.empty

    def reuse(*args, **kw):  # the allocator hands the same memory out again
        return memory if args and args[0] == total else empty(*args, **kw)

    torch.empty = reuse
    try:
        batch = GaussBatch(sc.n, sc.cameras, 16, -1, pair_capacity=1 << 20, device=dev)
    finally:
        torch.empty = empty
    assert batch.ws.data_ptr() == memory.data_ptr()
    got = gradients(batch)
    for k in want:
        scale = np.abs(want[k]).max()
        assert np.abs(got[k] - want[k]).max() <= 1e-5 * scale, k
