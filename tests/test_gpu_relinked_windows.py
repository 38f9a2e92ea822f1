"""Boundaries that do not hold, in windows that others follow: crowded movies
of blinking spots over several windows.  The segment behind such a boundary is
linked again from the true state, which then goes on to the next window; ids
and durations are the oracle's."""
import ctypes

import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200._params import trackpy_params
from test_gpu_link_stops import LINK_COLS, ctx, hook  # noqa: F401
from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


def blinking(frames, n, seed, side=96, seen=0.6, step=1.6):
    """Spots of width 1.3 that are there in some of the frames."""
    rng = np.random.default_rng(seed)
    pos = rng.uniform(8, side - 8, (n, 2))
    yy, xx = np.mgrid[0:side, 0:side]
    out = np.empty((frames, side, side), np.uint16)
    for t in range(frames):
        img = np.full((side, side), 100.0)
        for y, x in pos[rng.random(n) < seen]:
            img += 900.0 * np.exp(-((yy - y) ** 2 + (xx - x) ** 2) / (2 * 1.3 ** 2))
        out[t] = rng.poisson(img)
        pos = np.clip(pos + rng.normal(0, step, pos.shape), 8, side - 8)
    return out


@pytest.mark.parametrize("memory,seed,frames", [(0, 0, 290), (1, 1, 290), (3, 0, 290), (3, 2, 290), (3, 0, 400)])
def test_relinked_before_the_last_window(oracle, ctx, memory, seed, frames):
    f = blinking(frames, 40, seed)
    kw = dict(minmass=300.0, separation=6, search_range=9.0, memory=memory)
    tab = oracle.batch(trackpy_params(7, **kw), f.astype(np.float32))
    assert_same(gt.batch(f, 7, tqdm=False, **kw), tab, LINK_COLS)
    n = (ctypes.c_uint32(), ctypes.c_uint32())
    P = ctypes.POINTER(ctypes.c_uint32)
    ctx.check(hook("gt__relinked_segments", P, P)(ctx.handle, ctypes.byref(n[0]), ctypes.byref(n[1])))
    if memory:      # without memory a boundary's state is its detections alone, and always holds
        assert n[0].value > 0
    else:
        assert n[0].value == n[1].value == 0
