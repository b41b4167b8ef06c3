"""The rounding error of the weight gradients of the proposal network's third convolution, on a
network whose activations and gradients are known exactly: copying convolutions before it, a last
convolution and output weights of small integers, and a logit so low that the gradient of the
loss is -1/n."""
import numpy as np
import pytest

from cistem_downstream_bah_b200 import proposal as PR
from tests.test_gpu_proposal import _layer_slices

pytestmark = pytest.mark.gpu
F32 = np.float32


def _pool(a):
    """2 x 2 maxima and the first place of each (0..3)."""
    n, c, h, _ = a.shape
    w = a.reshape(n, c, h // 2, 2, h // 2, 2).transpose(0, 1, 2, 4, 3, 5).reshape(n, c, h // 2, h // 2, 4)
    return w.max(-1), w.argmax(-1)


def _padded(a):
    return np.pad(a, ((0, 0), (0, 0), (1, 1), (1, 1)))


def _conv(a, w):
    """3 x 3 convolution (cross-correlation), zero padding, in FP64."""
    n, _, h, _ = a.shape
    p = _padded(a)
    return sum(np.einsum("ncyx,oc->noyx", p[:, :, ky:ky + h, kx:kx + h], w[:, :, ky, kx], optimize=True)
               for ky in range(3) for kx in range(3))


def _case(tile, n, seed):
    rng = np.random.default_rng(seed)
    cin = PR.FEATURES
    sl = _layer_slices(cin)
    params = np.zeros(sl["b5"].stop, F32)
    for name, ci, co in (("w1", cin, 32), ("w2", 32, 64), ("w3", 64, 128)):
        w = params[sl[name]].reshape(co, ci, 3, 3)
        w[np.arange(co), np.arange(co) % ci, 1, 1] = 1   # channel o is channel o mod ci
    w4 = rng.integers(-2, 3, (128, 128, 3, 3)).astype(F32)
    w5 = rng.integers(1, 9, 128).astype(F32) * rng.choice([-1, 1], 128).astype(F32)
    params[sl["w4"]] = w4.ravel()
    params[sl["w5"]].reshape(4, 128)[0] = w5 / 8
    params[sl["b5"]][0] = -1e6
    x = rng.standard_normal((n, cin, tile, tile)).astype(F32)
    q = np.maximum(x, 0)
    for co in (32, 64):
        q = _pool(q[:, np.arange(co) % q.shape[1]])[0]
    a3 = q[:, np.arange(128) % 64]
    q3, place = _pool(a3)
    a4 = _conv(q3.astype(np.float64), w4.astype(np.float64)).reshape(n, 128, -1)
    top = np.partition(a4, -2, -1)[:, :, -2:]
    assert (top[:, :, 1] - top[:, :, 0]).min() > 1e-5   # no maximum is decided by rounding
    d4 = np.zeros_like(a4)
    np.put_along_axis(d4, a4.argmax(-1)[:, :, None], np.where(a4.max(-1) > 0, -w5.astype(np.float64) / 8 / n, 0)[:, :, None], -1)
    d4 = d4.reshape(q3.shape)
    dq3 = _conv(d4, w4.transpose(1, 0, 2, 3)[:, :, ::-1, ::-1].astype(np.float64))
    assert np.array_equal(dq3, dq3.astype(F32))   # multiples of 1 / (8 n)
    h = q3.shape[-1]
    d3 = (np.arange(4) == place[..., None]) * dq3[..., None]
    d3 = d3.reshape(n, 128, h, h, 2, 2).transpose(0, 1, 2, 4, 3, 5).reshape(a3.shape) * (a3 > 0)
    return params, x, q, d3.astype(F32)


def _threads_sum(g, x, threads=256):
    """FP32 sums over the last axis of g x (multiply-adds, zeros of g left out): one chain per
    thread over every 256th product, a tree over 32 threads, then the warps in order."""
    prod = g.astype(np.float64) * x
    k = prod.shape[-1] // threads
    prod = prod.reshape(*prod.shape[:-1], k, threads)
    s = np.zeros(prod.shape[:-2] + (threads,), F32)
    for i in range(k):
        s = (s + prod[..., i, :]).astype(F32)
    s = s.reshape(*s.shape[:-1], threads // 32, 32)
    while s.shape[-1] > 1:
        s = s[..., :s.shape[-1] // 2] + s[..., s.shape[-1] // 2:]
    total = np.zeros(s.shape[:-2], F32)
    for w in range(threads // 32):
        total = total + s[..., w, 0]
    return total


@pytest.mark.parametrize("tile,n", [(64, 128), (32, 128), (64, 32)])
def test_weight_gradients_are_no_less_accurate_than_sums_by_thread(tile, n):
    params, x, q2, d3 = _case(tile, n, seed=tile + n)
    net = PR.ProposalNet(PR.FEATURES, tile, max_batch=n)
    try:
        net.set_params(params)
        lab = np.tile(np.array([[1, 0, 0, 1]], F32), (n, 1))
        _, g = net.gradients(x, lab, pos_weight=1.0, dir_weight=0.0)
    finally:
        net.close()
    dw = g[_layer_slices(PR.FEATURES)["w3"]].reshape(128, 64, 3, 3)
    h = q2.shape[-1]
    p = _padded(q2)
    o, i = np.arange(0, 128, 8), np.arange(0, 64, 8)
    gs = d3[:, o].transpose(1, 0, 2, 3).reshape(len(o), 1, -1)
    err, bound = [], []
    for ky in range(3):
        for kx in range(3):
            xs = p[:, i, ky:ky + h, kx:kx + h].transpose(1, 0, 2, 3).reshape(1, len(i), -1)
            exact = (gs.astype(np.float64) * xs).sum(-1)
            err.append(dw[o][:, i, ky, kx] - exact)
            bound.append(_threads_sum(gs, xs) - exact)
            scale = np.sqrt((exact * exact).mean())
            assert np.abs(err[-1]).max() <= 1e-5 * scale   # the same network
    err, bound = np.array(err), np.array(bound)
    # a tenth for the order of additions, which the atomics leave open
    assert np.sqrt((err * err).mean()) <= 1.1 * np.sqrt((bound * bound).mean())
