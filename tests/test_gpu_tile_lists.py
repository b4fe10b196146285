"""Tile lists at the sizes where their kernels change course: superblock
sides of 1, 2, 4 and 8 tiles, superblock lists around the 1024-entry segments
they are split in.  Oracle: the reference's order, bit for bit."""
import numpy as np
import pytest

from dsplat import cudarc
from gpu_util import F, T, U32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 1023, 1024, 1025, 3100])
@pytest.mark.parametrize("side", [64, 250, 512, 1024])  # 8x8 tiles: superblocks of 1, 2, 4 and 8 tiles per side
def test_segmented_lists(orc, dev, side, n):
    rng = np.random.default_rng(n + side)
    xyd = np.empty((n, 3), np.float32)
    xyd[:, :2] = rng.uniform(0, 100, (n, 2))
    xyd[:, 2] = rng.integers(-4, 5, n) / 4.0  # depth ties
    half = rng.uniform(0, 70, (n, 2)).astype(np.float32)
    half[rng.random(n) < 0.3] = 200.0  # boxes that hold the corner's superblocks whole
    aabb = np.concatenate([xyd[:, :2] - half, xyd[:, :2] + half], axis=1).astype(np.float32)
    t2i, i2p, keys = cudarc.splat_gauss_tile2idx_idx2pnt(None, (side, side - 3), 8, T(xyd, dev), T(aabb, dev),
                                                         with_keys=True)
    o_t, o_i, o_k = orc.tile2pnt(xyd, aabb, side, side - 3, 8)
    assert np.array_equal(U32(t2i), o_t)
    assert np.array_equal(U32(i2p), o_i)
    assert np.array_equal(F(keys).view(np.uint64), o_k)


@pytest.mark.parametrize("n", [512, 513, 4095, 4097, 8192, 8193, 131072, 131073])
def test_sort_forms(orc, dev, n):
    """Around the limits between the sort in one block (512 and 1024 threads),
    the one whose blocks sum the digit counts and the one that scans them;
    equal depths, points without a tile and depths below -1 among them."""
    rng = np.random.default_rng(n)
    xyd = np.empty((n, 3), np.float32)
    xyd[:, :2] = rng.uniform(-30, 130, (n, 2))
    xyd[:, 2] = np.where(rng.random(n) < 0.5, rng.uniform(-1.2, 1.2, n), rng.integers(-4, 5, n) / 4.0)
    half = rng.uniform(0, 3, (n, 2)).astype(np.float32)
    aabb = np.concatenate([xyd[:, :2] - half, xyd[:, :2] + half], axis=1).astype(np.float32)
    t2i, i2p, keys = cudarc.splat_gauss_tile2idx_idx2pnt(None, (100, 90), 16, T(xyd, dev), T(aabb, dev), with_keys=True)
    o_t, o_i, o_k = orc.tile2pnt(xyd, aabb, 100, 90, 16)
    assert np.array_equal(U32(t2i), o_t)
    assert np.array_equal(U32(i2p), o_i)
    assert np.array_equal(F(keys).view(np.uint64), o_k)


@pytest.mark.parametrize("n", [524288, 524289, 606208, 606209, 1048576, 1048577])
def test_sort_tiles(orc, dev, n):
    """Around the limits between tiles of 2048 and 4096 keys and between blocks
    that sum their segment's counts and the scan of them; equal depths among
    the keys."""
    rng = np.random.default_rng(n)
    xyd = np.empty((n, 3), np.float32)
    xyd[:, :2] = rng.uniform(-30, 130, (n, 2))
    xyd[:, 2] = np.where(rng.random(n) < 0.5, rng.uniform(-1.2, 1.2, n), rng.integers(-4, 5, n) / 4.0)
    aabb = np.concatenate([xyd[:, :2] - 1, xyd[:, :2] + 1], axis=1).astype(np.float32)
    t2i, i2p = cudarc.splat_gauss_tile2idx_idx2pnt(None, (100, 90), 16, T(xyd, dev), T(aabb, dev))
    o_t, o_i, _ = orc.tile2pnt(xyd, aabb, 100, 90, 16)
    assert np.array_equal(U32(t2i), o_t)
    assert np.array_equal(U32(i2p), o_i)
