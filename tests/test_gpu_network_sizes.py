"""The proposal network's convolution and weight-gradient kernels at every tile
edge and at batches that do not fill a step of the weight gradient, against the
FP64 oracle; and an input that is not a number, which the ReLU masks."""
import numpy as np
import pytest

from cistem_downstream_bah_b200 import proposal as PR
from oracle import proposal as OP
from tests.test_gpu_proposal import _labels, _layer_slices

pytestmark = pytest.mark.gpu


def _gradients(tile, n, x, lab, params):
    net = PR.ProposalNet(PR.FEATURES, tile, max_batch=n)
    try:
        net.set_params(params)
        return net.gradients(x, lab, pos_weight=2.0, dir_weight=0.5)
    finally:
        net.close()


@pytest.mark.parametrize("tile,n", [(16, 1), (16, 67), (32, 1), (32, 18), (64, 5), (128, 2)])
def test_gradients_at_every_tile_edge(tile, n):
    rng = np.random.default_rng(100 * tile + n)
    params = PR.init_params(PR.FEATURES, seed=tile)
    x = rng.standard_normal((n, PR.FEATURES, tile, tile)).astype(np.float32)
    lab = _labels(n, rng)
    loss, g = _gradients(tile, n, x, lab, params)
    rloss, rg = OP.gradients(params.astype(np.float64), x, lab, PR.FEATURES, 2.0, 0.5, bf16=True)
    assert abs(loss - rloss) <= 1e-4 * abs(rloss)
    for name, sl in _layer_slices(PR.FEATURES).items():
        # the bound of the oracle comparison: a max-pool near-tie may route a pixel differently in FP32
        assert np.linalg.norm(g[sl] - rg[sl]) <= 2e-3 * np.linalg.norm(rg[sl]) + 1e-7, name


def test_masked_input_leaves_gradients_finite():
    rng = np.random.default_rng(3)
    params = PR.init_params(PR.FEATURES, seed=3)
    x = rng.standard_normal((2, PR.FEATURES, 32, 32)).astype(np.float32)
    x[0, 2, 7, 9] = np.nan
    loss, g = _gradients(32, 2, x, _labels(2, rng), params)
    assert np.isfinite(loss) and np.isfinite(g).all()
