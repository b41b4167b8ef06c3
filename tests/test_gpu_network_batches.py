"""The proposal network at the numbers of tiles where a layer's convolution changes its form, and at
those that do not fill its blocks."""
import time

import numpy as np
import pytest

from cistem_downstream_bah_b200 import proposal as PR
from oracle import proposal as OP
from tests.test_gpu_proposal import _labels, _layer_slices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile,n", [(16, 2), (16, 17), (16, 37), (16, 38), (16, 288), (16, 321), (32, 3), (32, 74), (32, 83),
                                    (64, 37), (64, 38)])
def test_outputs_do_not_depend_on_the_number_of_tiles(tile, n):
    """Every output is one chain of multiply-adds in the same order in every form: equal bits."""
    rng = np.random.default_rng(tile + n)
    x = rng.standard_normal((n, PR.FEATURES, tile, tile)).astype(np.float32)
    net = PR.ProposalNet(PR.FEATURES, tile, max_batch=n)
    try:
        net.set_params(PR.init_params(PR.FEATURES, seed=5))
        out = net.forward(x)
        alone = np.concatenate([net.forward(x[i:i + 1]) for i in range(n)])
    finally:
        net.close()
    assert np.array_equal(out, alone)


@pytest.mark.parametrize("tile,n", [(16, 33), (16, 289), (32, 75), (64, 38)])
def test_gradients_match_oracle(tile, n):
    rng = np.random.default_rng(100 * tile + n)
    params = PR.init_params(PR.FEATURES, seed=tile)
    x = rng.standard_normal((n, PR.FEATURES, tile, tile)).astype(np.float32)
    lab = _labels(n, rng)
    net = PR.ProposalNet(PR.FEATURES, tile, max_batch=n)
    try:
        net.set_params(params)
        loss, g = net.gradients(x, lab, pos_weight=2.0, dir_weight=0.5)
    finally:
        net.close()
    rloss, rg = OP.gradients(params.astype(np.float64), x, lab, PR.FEATURES, 2.0, 0.5, bf16=True)
    assert abs(loss - rloss) <= 1e-4 * abs(rloss)
    for name, sl in _layer_slices(PR.FEATURES).items():
        # the bound of the oracle comparison: a max-pool near-tie may route a pixel differently in FP32
        assert np.linalg.norm(g[sl] - rg[sl]) <= 2e-3 * np.linalg.norm(rg[sl]) + 1e-7, name


def test_small_tiles_take_no_longer_than_large_ones():
    """Two tiles of 16 x 16 hold a sixteenth of the work of two of 64 x 64."""
    best = {}
    for tile in (16, 64):
        net = PR.ProposalNet(PR.FEATURES, tile, max_batch=2)
        try:
            net.set_params(PR.init_params(PR.FEATURES, seed=1))
            x = np.zeros((2, PR.FEATURES, tile, tile), np.float32)
            times = []
            for _ in range(200):
                t0 = time.perf_counter()
                net.forward(x)
                times.append(time.perf_counter() - t0)
            best[tile] = min(times)
        finally:
            net.close()
    assert best[16] <= 1.3 * best[64], best
