"""The batched projection at every colour degree, around the ends of its
blocks of 128 points: records, tile lists and images bit for bit against the
oracle."""
import pytest

from dsplat.gauss import GaussBatch
from gpu_util import params_of
from test_gpu_fused import _check_view, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 300])
@pytest.mark.parametrize("sh_deg", [-1, 0, 1, 2, 3])
def test_degrees(orc, dev, sh_deg, n):
    sc = _scene(sh_deg, n=n, seed=11)
    params = params_of(sc, dev)
    batch = GaussBatch(sc.n, sc.cameras, 8, sc.sh_degree, pair_capacity=1 << 16, device=dev)
    batch.ensure_capacity(params)
    batch.forward(params)
    for v in range(len(sc.cameras)):
        _check_view(orc, batch, sc, v, 8)
