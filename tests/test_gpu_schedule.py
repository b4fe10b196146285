"""The task schedule of the batched rasterisers: what it is formed from."""
import numpy as np
import pytest

from dsplat import scenes
from dsplat.gauss import GaussBatch
from gpu_util import F, params_of
from schedule_util import CONFIGS, heavy_items, item_cost, masks, set_blocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ts,ppl", CONFIGS)
def test_measured_cost_does_not_depend_on_the_shape(dev, ts, ppl):
    """An item's cost is the same walked in blocks or in whole tasks, so that
    the same inputs lead to the same schedule again."""
    sc = scenes.config0(seed=2, n=900, size=(133, 94))
    p = params_of(sc, dev)
    batch = GaussBatch(sc.n, sc.cameras, ts, -1, pair_capacity=1 << 16, device=dev, pixels_per_lane=ppl)
    batch.ensure_capacity(p)
    costs = []
    for blocks in masks(batch):
        set_blocks(batch, blocks)
        batch.forward(p)
        costs.append(F(item_cost(batch)).copy())
    assert costs[0].max() > 0
    assert np.array_equal(*costs)


def test_first_forward_on_a_workspace_ignores_what_it_held(dev):
    """The items' costs count once a forward has measured them: on a workspace
    full of anything else the schedule is that of the list lengths."""
    sc = scenes.config0(seed=8, n=1500, size=(1297, 1013))  # about 10,000 items that lead a task
    p = params_of(sc, dev)
    heavy = []
    for fill in (0, 0xff, 0x01):
        batch = GaussBatch(sc.n, sc.cameras, 8, -1, pair_capacity=1 << 18, device=dev)
        batch.ws.fill_(fill)
        batch.forward(p)
        heavy.append(heavy_items(batch))
        assert batch.status()[0] == 0
    assert 0 < heavy[0] < int(batch.layout.num_items)
    assert heavy == [heavy[0]] * 3
