"""Weight gradients at the edges of their 4 x 32 cell tiles (a single cell, a
tile less one, one more, several tiles a CTA) against the numpy oracle, to the
tolerance of the gradient test (BF16 roundings of near-tied activations), and
training twice from one state with and without kept buffers, bit for bit."""
import ctypes

import numpy as np
import pytest

from gpu_tracking_b200 import _ffi, learned
from oracle import cnn_oracle as co
from synth import video
from test_gpu_learned import random_net, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crop,B", [(4, 3), (12, 5), (124, 2), (128, 2), (132, 2), (20, 400)])
def test_gradients_over_tile_edges(crop, B):
    frames, truth = video(2, 140, 140, 40, seed=crop)
    net, p = random_net(3)
    mean, scale = float(frames.mean()), 1.0 / float(frames.std())
    net.set_normalization(mean, scale)
    lf = np.concatenate([np.full(len(t), k) for k, t in enumerate(truth)]).astype(np.int64)
    ly = np.concatenate(truth)[:, 0].astype(np.float32)
    lx = np.concatenate(truth)[:, 1].astype(np.float32)
    rng = np.random.default_rng(crop)
    at = (140 - crop) // 4
    crops = np.column_stack([rng.integers(0, 2, B), 4 * rng.integers(0, at + 1, B),
                             4 * rng.integers(0, at + 1, B)]).astype(np.int32)
    grad = np.zeros(co.num_params(), np.float32)
    loss = np.zeros(2, np.float32)
    P32, P64 = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_int64)
    ctx = _ffi.context(0)
    ctx.check(_ffi.lib().gt__proposal_loss_grad(
        ctx.handle, net.handle, ctypes.c_void_p(frames.ctypes.data), 0, *frames.shape, lf.ctypes.data_as(P64),
        ly.ctypes.data_as(P32), lx.ctypes.data_as(P32), len(lf), crops.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)),
        B, crop, 8.0, 1.0, grad.ctypes.data_as(P32), loss.ctypes.data_as(P32)))
    x = co.cells(frames, mean, scale, crops=crops, crop=crop)
    tmap = co.targets(lf, ly, lx, 2, 35, 35)
    tgt = np.stack([tmap[f, y // 4:y // 4 + crop // 4, c // 4:c // 4 + crop // 4] for f, y, c in crops])
    _, g = co.loss_grad(p, x, tgt, 8.0, 1.0)
    o = 0
    for l, (ci, cout) in enumerate(zip(co.CIN, co.COUT)):
        for n in (cout * ci * 9, cout):
            assert rel_err(grad[o:o + n], g[o:o + n]) < 3e-2, l
            o += n


def test_kept_buffers_change_nothing():
    frames, truth = video(3, 96, 96, 30, seed=8)
    labels = {"frame": np.concatenate([np.full(len(t), k) for k, t in enumerate(truth)]),
              "y": np.concatenate(truth)[:, 0], "x": np.concatenate(truth)[:, 1]}
    runs = []
    for _ in range(3):
        net = learned.ProposalNet(seed=2)
        net.set_normalization(100.0, 0.1)
        runs.append((net.train(frames, labels, steps=3, batch=8, crop=64), net.params))
    # a net that trains on larger, smaller and again larger crops reuses its buffers
    net = learned.ProposalNet(seed=2)
    net.set_normalization(100.0, 0.1)
    start = net.params
    net.train(frames, labels, steps=1, batch=16, crop=96)
    net.train(frames, labels, steps=1, batch=2, crop=8)
    fresh = learned.ProposalNet(seed=2)
    fresh.set_normalization(100.0, 0.1)
    fresh.train(frames, labels, steps=1, batch=16, crop=96)
    fresh.train(frames, labels, steps=1, batch=2, crop=8)
    assert np.array_equal(net.params, fresh.params) and not np.array_equal(net.params, start)
    for loss, params in runs[1:]:
        assert np.array_equal(loss, runs[0][0]) and np.array_equal(params, runs[0][1])
