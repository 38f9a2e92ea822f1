"""A call that fails leaves nothing behind for the next call on its thread
(CUDA keeps the last error per thread, and short calls run on the caller's)."""
import ctypes

import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200 import _ffi
from test_gpu_link_stops import hook

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("after", ["batch", "link", "train"])
def test_next_call_after_out_of_memory(after):
    from gpu_tracking_b200 import learned
    ctx = _ffi.context(0)
    f = np.random.default_rng(0).integers(50, 200, (40, 64, 64)).astype(np.uint16)
    r = np.array([[t, 5.0 + t, 5.0] for t in range(20)], np.float32)
    kw = dict(minmass=30.0, search_range=3.0, tqdm=False)
    want = gt.batch(f, 9, **kw)
    caps = hook("gt__set_link_window_caps", ctypes.c_int64, ctypes.c_int64)
    try:
        ctx.check(caps(ctx.handle, 0, 40 * 10 ** 9))   # 320 GB of edges
        with pytest.raises(_ffi.GpuTrackingError, match="memory"):
            gt.batch(f, 9, **kw)
    finally:
        ctx.check(caps(ctx.handle, 0, 0))
    if after == "batch":
        assert np.array_equal(gt.batch(f, 9, **kw).to_numpy(), want.to_numpy(), equal_nan=True)
    elif after == "link":
        assert np.array_equal(gt.link(r, 3.0), np.zeros(20))
    else:
        net = learned.ProposalNet(seed=0)
        net.train(f, want[["frame", "y", "x"]], steps=1, batch=2, crop=32)
