"""The rasterisers' two task shapes, 8x8 blocks (the longest walks of a batch,
every drop-in call) and whole tasks, at the edges of blocks and tiles and at
every tile size and pixels-per-lane choice; which items are walked in blocks is
up to the schedule here (test_gpu_loss.py, test_gpu_schedule.py and
test_gpu_nonfinite.py choose it).  Images, transmittances and stop positions bit
for bit against the oracle; gradients against its FP64 backward at the tolerance
of test_gpu_grad.py (rel 1e-3, floor 1e-2 of the largest component, 99.9% of the
components)."""
import numpy as np
import pytest
import torch

from dsplat import cudarc, scenes
from gpu_util import F, T
from test_gpu_grad import GROUPS, _close, _run

pytestmark = pytest.mark.gpu


def _check(orc, dev, n, size, ts, ppl):
    from dsplat import gauss
    sc = scenes.config0(seed=n + ts, n=n, size=size)
    target = np.random.default_rng(n).uniform(0, 1, (size[1], size[0], 3)).astype(np.float32)

    class Batch(gauss.GaussBatch):  # _run's batch with this pixels-per-lane choice
        def __init__(self, *a, **k):
            super().__init__(*a, pixels_per_lane=ppl, **k)

    import test_gpu_grad
    keep, test_gpu_grad.GaussBatch = test_gpu_grad.GaussBatch, Batch
    try:
        batch, g_gpu, S = _run(orc, dev, sc, target, ts)
    finally:
        test_gpu_grad.GaussBatch = keep
    cam = sc.cameras[0]
    xyd, conic, aabb, rgb = orc.fused_project(sc.means, sc.log_scales, sc.quats, sc.colors, -1, cam.mvp, cam.campos, *size)
    t2i, i2p, stop = batch.tile_lists(0)
    img, trans, last = orc.gauss_rasterize_tiled(*size, ts, t2i, i2p, xyd, conic, aabb, sc.opacity, rgb, nthreads=8)
    assert np.array_equal(F(batch.images()[0]), img)
    assert np.array_equal(F(batch.per_pixel("T")[0]), trans)
    assert np.array_equal(stop, last)
    loss = float(batch.slab_loss().double().sum())
    want = float(((img.astype(np.float64) - target) ** 2).sum())
    assert abs(loss - want) <= 1e-5 * want
    _, g64 = S.backward()
    for k in GROUPS:
        ref = g64[k].reshape(sc.n, -1)
        ok = _close(g_gpu[k], ref, np.abs(ref).max(), 1e-3, 1e-2)
        assert ok.mean() > 0.999, (k, ok.mean())


@pytest.mark.parametrize("ts", [8, 16, 32])
@pytest.mark.parametrize("size", [(1, 1), (7, 9), (8, 8), (9, 17), (33, 24), (100, 70)])
def test_blocks(orc, dev, size, ts):
    _check(orc, dev, 400, size, ts, 0)


@pytest.mark.parametrize("ts,ppl", [(8, 1), (8, 2), (16, 2), (16, 4), (16, 8), (32, 4), (32, 8)])
def test_large_view(orc, dev, ts, ppl):
    _check(orc, dev, 1500, (1297, 1013), ts, ppl)


@pytest.mark.parametrize("ts", [8, 16, 32])
def test_infinite_colour_stays_in_its_box(orc, dev, ts):
    sc = scenes.config0(seed=5, n=300, size=(90, 60))
    cam = sc.cameras[0]
    rgb = sc.colors.copy()
    rgb[::7] = np.inf
    rgb[3::11, 1] = np.nan
    xyd, conic, aabb = orc.gauss_project(sc.means, sc.quats, sc.scales, cam.mvp, 90, 60)
    t2i, i2p, _ = orc.tile2pnt(xyd, aabb, 90, 60, ts)
    want, _, _ = orc.gauss_rasterize_tiled(90, 60, ts, t2i, i2p, xyd, conic, aabb, sc.opacity, rgb)
    img = torch.zeros((60, 90, 3), device=dev)
    cudarc.splat_gauss_rasterize_pnt2splat2(None, (90, 60), img, T(xyd, dev), T(conic, dev), T(aabb, dev),
                                            T(sc.opacity, dev), T(rgb, dev), ts, T(t2i.view(np.int32), dev),
                                            T(i2p.view(np.int32), dev))
    assert np.isfinite(want).any() and not np.isfinite(want).all()
    assert np.array_equal(F(img), want, equal_nan=True)
