"""Training's working memory belongs to the context: networks that were trained
hold their parameters alone, a fresh one trains in what the last one used, and
several threads train at once."""
import threading

import numpy as np
import pytest

from gpu_tracking_b200 import learned
from synth import video

pytestmark = pytest.mark.gpu

STEPS = dict(steps=2, batch=256, crop=96)   # buffers of some 70 MB


@pytest.fixture(scope="module")
def data():
    f, truth = video(4, 96, 128, n_spots=12, seed=5)
    rows = np.concatenate([np.column_stack([np.full(len(t), k), t]) for k, t in enumerate(truth)])
    return f, dict(zip(("frame", "y", "x"), rows.T))


def trained(data, seed):
    net = learned.ProposalNet(seed=seed)
    losses = net.train(data[0], data[1], **STEPS)
    return net, net.params.copy(), np.asarray(losses)


def used():
    import torch
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_networks_hold_no_working_memory(data):
    nets = [trained(data, 0)]
    before = used()
    nets += [trained(data, s) for s in range(1, 9)]
    assert used() - before < 64 << 20


def test_same_weights_whatever_was_left_behind(data):
    _, want, losses = trained(data, 3)
    other = learned.ProposalNet(seed=1)
    other.train(data[0], data[1], steps=1, batch=7, crop=32)     # other sizes in between
    other.train(data[0], data[1], steps=1, batch=96, crop=96)
    _, got, again = trained(data, 3)
    assert np.array_equal(got, want) and np.array_equal(again, losses)


def test_threads_train_different_networks(data):
    want = {s: trained(data, s)[1] for s in range(4)}
    got = {}

    def work(s):
        for _ in range(3):
            got[s] = trained(data, s)[1]

    th = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert all(np.array_equal(got[s], want[s]) for s in range(4))
