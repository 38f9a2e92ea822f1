"""The pool of pinned result blocks: bounded, a block is never in two results
at once, pinned only for sizes of which many results were dropped; and on a GPU the
pinned and the pageable way of a table, and of frames large enough for the
upload lanes, give the same values."""
import gc
import threading

import numpy as np
import pytest

from gpu_tracking_b200 import _ffi


class FakeLib:
    def __init__(self):
        self.live = {}
        self.most = 0

    def gt_host_alloc(self, size):
        a = np.zeros(size, np.uint8)
        self.live[a.ctypes.data] = a
        self.most = max(self.most, sum(len(x) for x in self.live.values()))
        return a.ctypes.data

    def gt_host_free(self, address):
        del self.live[address]


@pytest.fixture
def fake(monkeypatch):
    lib = FakeLib()
    monkeypatch.setattr(_ffi, "lib", lambda: lib)
    return lib


def test_kept_results_are_never_pinned(fake):
    pool = _ffi.ResultPool(limit=8 << 20)
    kept = [np.asarray(pool.take(1 << 20)) for _ in range(5)]
    assert not fake.live and len({a.ctypes.data for a in kept}) == 5


def test_dropped_results_are_pinned_and_reused(fake):
    pool = _ffi.ResultPool(limit=8 << 20)
    assert pool.earned(2 << 20) < pool.earned(64 << 20)
    for k in range(pool.earned(2 << 20) + 6):
        assert bool(fake.live) == (k > pool.earned(2 << 20))
        a = np.asarray(pool.take(1 << 20))[: 1 << 20].view(np.float64)[7:]   # views keep the block
        a[:] = 3.0
        del a
        gc.collect()
    assert len(fake.live) == 1
    b = pool.take(1 << 20)
    v = np.asarray(b)[:64]
    address = b.address
    del b
    gc.collect()
    assert np.asarray(pool.take(1 << 20)).ctypes.data != address   # v still holds it
    del v
    gc.collect()
    pool.trim()
    assert not fake.live


def test_ordinary_blocks_are_reused_within_the_limit(fake):
    pool = _ffi.ResultPool(limit=8 << 20)
    pool.PIN_AFTER = 30
    held = [pool.take((2 << 20) - 1) for _ in range(6)]
    addresses = {b.address for b in held}
    del held
    gc.collect()
    assert pool._kept == 8 << 20
    again = [pool.take((2 << 20) - 1) for _ in range(4)]
    assert {b.address for b in again} <= addresses and pool._kept == 0
    for _ in range(2 * pool.PIN_AFTER):
        pool.take(3 << 20)               # a block of half the limit: never pinned
        gc.collect()
    assert not fake.live


def test_limit_and_threads(fake):
    pool = _ffi.ResultPool(limit=4 << 20)
    wrong = []

    def work(seed):
        rng = np.random.default_rng(seed)
        held = []
        for k in range(200):
            n = int(rng.integers(1, 1 << 20))
            a = np.asarray(pool.take(n))[:n]
            a[:] = seed
            held.append(a)
            if len(held) > 3:
                b = held.pop(int(rng.integers(0, 3)))
                if not (b == seed).all():
                    wrong.append(seed)

    th = [threading.Thread(target=work, args=(s,)) for s in range(1, 5)]
    [t.start() for t in th]
    [t.join() for t in th]
    gc.collect()
    assert not wrong and fake.most <= 4 << 20


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.uint8, np.float32])
def test_table_and_upload_ways_agree(dtype, monkeypatch):
    import pandas as pd
    import torch

    import gpu_tracking_b200 as gt
    from synth import video
    f, _ = video(150, 187, 211, n_spots=25, seed=3, dtype=dtype, amp_mu=np.log(90.0), bg=40.0,
                 read_noise=3.0 if dtype == np.float32 else None)
    assert f.nbytes > 5 << 20            # several slots of every lane
    kw = dict(minmass=60.0, search_range=4.0, memory=1, tqdm=False)
    monkeypatch.setattr(_ffi.ResultPool, "PIN_AFTER", 1)
    first = gt.batch(f, 7, **kw)         # pageable result, pageable frames
    copy = first.copy(deep=True)
    dropped = gt.batch(f, 7, **kw)
    del dropped
    for _ in range(3):                   # pinned result
        again = gt.batch(torch.from_numpy(f).cuda(), 7, **kw)
        pd.testing.assert_frame_equal(again, copy, check_exact=True)
    pd.testing.assert_frame_equal(first, copy, check_exact=True)
    assert len(gt.batch(f, 7, minmass=1e9, tqdm=False)) == 0
