"""The superblock scatter that does not stage its entries in shared memory:
views whose superblock counters leave no room for them."""
import pytest

from dsplat import scenes
from dsplat.gauss import GaussBatch
from gpu_util import params_of
from test_gpu_fused import _check_view

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [700, 9000])  # 2 chunks of 512 ranks and 24
def test_unstaged_scatter(orc, dev, n):
    """3328x3328 in 8x8 tiles: 52x52 superblocks.  The staged form needs 45,064
    bytes and 24 per superblock, 109,964 here, and is used up to 102,400."""
    sc = scenes.config0(seed=n, n=n, size=(64, 64))
    sc.cameras = [scenes.Camera.look_at_origin((0.1, 0.3, -3.0), 3328, 3328)]
    p = params_of(sc, dev)
    batch = GaussBatch(sc.n, sc.cameras, 8, sc.sh_degree, pair_capacity=1 << 21, device=dev)
    assert int(batch.layout.sb_log2[0]) == 3 and int(batch.layout.num_sb) == 52 * 52
    batch.ensure_capacity(p)
    assert batch.status()[0] == 0
    _check_view(orc, batch, sc, 0, 8)
