"""Weight gradients of the proposal network for gradients that are infinite at a map's border."""
import numpy as np
import pytest

from cistem_downstream_bah_b200 import proposal as PR
from tests.test_gpu_proposal import _layer_slices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [16, 32])
def test_infinite_gradient_leaves_the_taps_outside_the_map_alone(tile):
    rng = np.random.default_rng(tile)
    params = PR.init_params(PR.FEATURES, seed=tile)
    x = rng.standard_normal((1, PR.FEATURES, tile, tile)).astype(np.float32)
    net = PR.ProposalNet(PR.FEATURES, tile, max_batch=1)
    try:
        net.set_params(params)
        # an infinite weight of the positives: the gradient of every active channel of the last
        # convolution is infinite at one pixel, its maximum, and zero elsewhere
        _, g = net.gradients(x, np.array([[1, 0, 0, 1]], np.float32), pos_weight=np.inf, dir_weight=0.0)
    finally:
        net.close()
    w4 = g[_layer_slices(PR.FEATURES)["w4"]].reshape(128, 128, 9)
    active = ~np.isfinite(w4).all((1, 2))   # output channels
    assert active.any()
    if tile == 16:   # 2 x 2 maps: five of the nine taps lie outside, whichever pixel it is
        assert (np.isfinite(w4).sum(-1) >= 5).all()
    else:            # 4 x 4 maps: three or five lie outside where the pixel is at the border
        untouched = (w4[active] == 0).all(1).sum(-1)
        assert set(untouched) <= {0, 3, 5} and (untouched > 0).any()
