"""The partial L2 losses of the batched forward (slab_loss): every slot is
written, whatever shape an item is walked in."""
import numpy as np
import pytest
import torch

from dsplat import scenes
from dsplat.gauss import GaussBatch
from gpu_util import F, params_of
from schedule_util import CONFIGS, heavy_items, leaders, masks, set_blocks

pytestmark = pytest.mark.gpu


def _batch(dev, size, ts, ppl, n=400):
    sc = scenes.config0(seed=n + ts, n=n, size=size)
    p = params_of(sc, dev)
    batch = GaussBatch(sc.n, sc.cameras, ts, -1, pair_capacity=1 << 16, device=dev, pixels_per_lane=ppl)
    batch.ensure_capacity(p)
    return batch, p, torch.rand(size[0] * size[1] * 3, device=dev)


@pytest.mark.parametrize("ts,ppl", CONFIGS)
@pytest.mark.parametrize("size", [(7, 9), (33, 24), (100, 70)])
def test_every_slot_is_written(dev, size, ts, ppl):
    """NaN in the slots before the forward; their sum against the images'
    float64 loss.  Tolerance: a slot sums at most 256 pixels' three squares in
    at most 40 roundings, 40 * 2^-24 < 1e-5 of a sum of non-negative terms."""
    batch, p, target = _batch(dev, size, ts, ppl)
    for blocks in masks(batch):
        set_blocks(batch, blocks)
        batch.slab_loss().fill_(float("nan"))
        batch.forward(p, target=target)
        assert heavy_items(batch) == int((blocks & leaders(batch)).sum())
        want = float(((batch.out_rgb.double() - target.double()) ** 2).sum())
        assert abs(float(batch.slab_loss().double().sum()) - want) <= 1e-5 * want


@pytest.mark.parametrize("ts,ppl", CONFIGS)
def test_loss_does_not_depend_on_the_schedule(dev, ts, ppl):
    """The same bits in every slot, whichever items are walked in blocks."""
    batch, p, target = _batch(dev, (133, 94), ts, ppl)
    seen = []
    for k in range(6):
        set_blocks(batch, masks(batch)[k % 2])
        batch.forward(p, target=target)
        seen.append(F(batch.slab_loss()).view(np.uint32).copy())
    for s in seen[1:]:
        assert np.array_equal(s, seen[0])
