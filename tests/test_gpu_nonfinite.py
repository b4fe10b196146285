"""Parameters, upstream gradients and conics that are not finite, or whose
inverse is not: what they may not reach."""
import numpy as np
import pytest
import torch

from dsplat import scenes
from dsplat.gauss import GaussBatch
from gpu_util import F, params_of
from schedule_util import CONFIGS, masks, set_blocks

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
