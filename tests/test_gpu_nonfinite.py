"""Parameters, upstream gradients and conics that are not finite, or whose
inverse is not: what they may not reach."""
import os

import numpy as np
import pytest
import torch

from dsplat import scenes
from dsplat.gauss import GaussBatch
from gpu_util import F, params_of
from schedule_util import CONFIGS, masks, odd, set_blocks

pytestmark = pytest.mark.gpu
GROUPS = ["means", "log_scales", "quats", "opacity", "colors"]


def test_zero_gradient_through_a_needle_is_zero(dev):
    """Needles whose covariance determinant is 0 or squares to 0 in float32:
    the forward holds their eigenvalues, and an upstream gradient of exactly 0
    gives them gradients of exactly 0."""
    sc = scenes.config0(seed=3, n=2000, size=(120, 90))
    sc.log_scales = np.tile(np.log(np.array([[0.1, 1e-5, 1e-5]], np.float32)), (sc.n, 1)).astype(np.float32)
    p = params_of(sc, dev)
    batch = GaussBatch(sc.n, sc.cameras, 16, -1, pair_capacity=1 << 18, device=dev)
    batch.ensure_capacity(p)
    assert batch.out_rgb.abs().max() > 0
    grads = {k: torch.zeros_like(v) for k, v in p.items()}
    batch.backward(p, grads, torch.zeros_like(batch.out_rgb))
    for k in GROUPS:
        assert not F(grads[k]).any(), k  # NaN counts as non-zero


def _pixel_scene(w=48, h=40):
    """One Gaussian per pixel, its box inside the pixel; a random half of them far, the others near."""
    rng = np.random.default_rng(9)
    n = w * h
    far = rng.random(n) < 0.5
    y, x = np.divmod(np.arange(n), w)
    means = np.stack([(x + 0.5) * 2 / w - 1, 1 - (y + 0.5) * 2 / h, np.where(far, -0.5, 0.5)], 1).astype(np.float32)
    ls = np.full((n, 3), np.log(0.1 / max(w, h)), np.float32)
    quats = np.tile(np.array([[0, 0, 0, 1]], np.float32), (n, 1))
    cam = scenes.Camera(w, h, np.eye(4, dtype=np.float32).reshape(16), np.zeros(3, np.float32))
    sc = scenes.GaussScene(means, ls, quats, np.full(n, 0.5, np.float32), rng.uniform(0, 1, (n, 3)).astype(np.float32),
                           -1, [cam], 8)
    return sc, far


@pytest.mark.parametrize("ts,ppl", CONFIGS)
@pytest.mark.parametrize("what", ["inf colour", "nan colour", "inf opacity", "nan opacity", "nan upstream"])
def test_backward_keeps_it_in_its_pixels(dev, ts, ppl, what):
    """Half of the pixels hold something that is not finite; the Gaussians of
    the other pixels get the gradients that they get without it."""
    sc, far = _pixel_scene()
    up = np.random.default_rng(4).uniform(-1, 1, (sc.n, 3)).astype(np.float32)
    results = []
    for odd in (False, True):
        p = params_of(sc, dev)
        grad_rgb = torch.from_numpy(up).to(dev)
        sel = torch.from_numpy(far).to(dev)
        if odd:
            value = float(what.split()[0])
            (p["colors"] if "colour" in what else p["opacity"] if "opacity" in what else grad_rgb)[sel] = value
        batch = GaussBatch(sc.n, sc.cameras, ts, -1, pair_capacity=1 << 16, device=dev, pixels_per_lane=ppl)
        batch.ensure_capacity(p)
        res = []
        for blocks in masks(batch):
            set_blocks(batch, blocks)
            batch.forward(p)
            grads = {k: torch.zeros_like(v) for k, v in p.items()}
            batch.backward(p, grads, grad_rgb.reshape(-1))
            res.append({k: F(grads[k])[~far] for k in GROUPS})
        results.append(res)
    for a, b in zip(*results):
        assert np.abs(a["colors"]).min() > 0
        for k in GROUPS:
            assert np.isfinite(a[k]).all() and np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("ts,ppl", CONFIGS)
def test_batched_image_keeps_odd_colours_in_their_boxes(orc, dev, ts, ppl):
    """Infinite and NaN colours, every item walked in both shapes: the
    oracle's image, bit for bit."""
    sc = scenes.config0(seed=5, n=300, size=(90, 60))
    sc.colors[::7] = np.inf
    sc.colors[3::11, 1] = np.nan
    cam = sc.cameras[0]
    p = params_of(sc, dev)
    batch = GaussBatch(sc.n, sc.cameras, ts, -1, pair_capacity=1 << 16, device=dev, pixels_per_lane=ppl)
    batch.ensure_capacity(p)
    xyd, conic, aabb, rgb = orc.fused_project(sc.means, sc.log_scales, sc.quats, sc.colors, -1, cam.mvp, cam.campos, 90, 60)
    t2i, i2p, _ = orc.tile2pnt(xyd, aabb, 90, 60, ts)
    want, _, _ = orc.gauss_rasterize_tiled(90, 60, ts, t2i, i2p, xyd, conic, aabb, sc.opacity, rgb)
    assert np.isfinite(want).any() and not np.isfinite(want).all()
    for blocks in masks(batch):
        set_blocks(batch, blocks)
        batch.forward(p)
        assert np.array_equal(F(batch.images()[0]), want, equal_nan=True)


def test_a_capture_is_not_odd(dev):
    """The slower form of the backward is for values that are not finite: the
    thin conics of a capture and an ordinary loss stay with the other."""
    from dsplat.render_ply import load_scene
    cams = scenes.sphere_cameras(np.random.default_rng(7), 8, 3.0, [(640, 480)])
    sc = load_scene(os.path.join(os.path.dirname(__file__), "golden", "bulba_subset.ply"), cams)
    p = params_of(sc, dev)
    batch = GaussBatch(sc.n, cams, 8, 3, pair_capacity=1 << 20, device=dev)
    batch.ensure_capacity(p)
    target = torch.rand(int(batch.layout.num_pix) * 3, device=dev)
    batch.forward(p, target=target)
    assert not odd(batch)
    target[7] = float("nan")
    batch.forward(p, target=target)
    assert odd(batch)
    batch.forward(p)
    assert not odd(batch)
    p["opacity"][5] = float("inf")
    batch.forward(p)
    assert odd(batch)
