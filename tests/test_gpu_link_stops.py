"""A linker that stops in the middle of a call.

A window's list kernels raise the overflow flag while the linker of the window
before still runs, and the first segment of a window raises the edge flag while
the window's other segments run.  Every CTA must take one decision about such a
flag for all of its threads; the call then links the whole video, and ids and
durations are the oracle's.
"""
import ctypes

import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200 import _ffi
from gpu_tracking_b200._params import trackpy_params
from synth import video
from test_gpu_parity import ALL_TP, assert_same

pytestmark = pytest.mark.gpu

LINK_COLS = ALL_TP + ["particle", "duration"]
RADIUS = 6.0


def hook(name, *argtypes):
    f = getattr(_ffi.lib(), name)
    f.argtypes = [ctypes.c_void_p, *argtypes]
    f.restype = ctypes.c_int32
    return f


@pytest.fixture
def ctx(monkeypatch):
    """A context of its own: capacities and buffers of no other test's."""
    c = _ffi.Context(0)
    monkeypatch.setitem(_ffi._contexts, 0, c)
    yield c
    c.close()


def caps(ctx):
    out = (ctypes.c_int64(), ctypes.c_int64())
    P = ctypes.POINTER(ctypes.c_int64)
    ctx.check(hook("gt__get_link_window_caps", P, P)(ctx.handle, ctypes.byref(out[0]), ctypes.byref(out[1])))
    return out[0].value, out[1].value


def movie(parts):
    """Frames of (count, spots) one after another."""
    return np.concatenate([video(n, 64, 64, spots, seed=70 + k, D=0.5)[0] for k, (n, spots) in enumerate(parts)])


def entries(df, frames, memory):
    """Backward neighbours of the points of `frames`, per frame."""
    at = {t: g[["y", "x"]].to_numpy() for t, g in df.groupby("frame")}
    out = []
    for t in frames:
        n = 0
        for k in range(1, memory + 2):
            if t in at and t - k in at:
                d = at[t][:, None] - at[t - k][None]
                n += int(((d ** 2).sum(2) <= RADIUS ** 2).sum())
        out.append(n)
    return np.array(out)


def run_small(ctx, f, memory, list_entries, edges, oracle):
    """The call with small window buffers equals the oracle; returns the buffers it ends with."""
    kw = dict(minmass=300.0, search_range=RADIUS, memory=memory)
    tab = oracle.batch(trackpy_params(9, **kw), f.astype(np.float32))
    set_caps = hook("gt__set_link_window_caps", ctypes.c_int64, ctypes.c_int64)
    try:
        for _ in range(5):
            ctx.check(set_caps(ctx.handle, list_entries, edges))
            assert_same(gt.batch(f, 9, tqdm=False, **kw), tab, LINK_COLS)
            now = caps(ctx)
    finally:
        ctx.check(set_caps(ctx.handle, 0, 0))
    assert_same(gt.batch(f, 9, tqdm=False, **kw), tab, LINK_COLS)
    return now


@pytest.mark.parametrize("memory", [0, 2, 17])   # 17: the sequential kernel
def test_lists_overflow_after_the_first_window(oracle, ctx, memory):
    f = movie([(140, 3), (160, 14)])
    df = gt.batch(f, 9, minmass=300.0, tqdm=False)
    e = entries(df, range(300), memory)
    room = int(e[:128].sum()) + 64
    # windows of 128 frames; the second one's lists go back over memory + 1 frames more
    assert e[128:256].sum() > 2 * room
    assert run_small(ctx, f, memory, room, 1 << 20, oracle) == (4 * room, 1 << 20)


@pytest.mark.parametrize("memory", [0, 1, 3])
def test_first_segment_stops_beside_others(oracle, ctx, memory):
    f = movie([(2, 16), (118, 2)])
    df = gt.batch(f, 9, minmass=300.0, tqdm=False)
    e = entries(df, range(120), memory)
    room = int(e[memory + 3:].max())
    assert e[1] > room
    assert run_small(ctx, f, memory, 1 << 20, room, oracle) == (1 << 20, 4 * room)


def grids(frames, dense):
    """Frames of noise, those of `dense` with a grid of 100 spots."""
    rng = np.random.default_rng(1)
    yy, xx = np.mgrid[0:240, 0:240]
    spots = sum(900.0 * np.exp(-((yy - y) ** 2 + (xx - x) ** 2) / 4.5)
                for y in range(12, 240, 24) for x in range(12, 240, 24))
    f = rng.poisson(100.0, (frames, 240, 240))
    f[list(dense)] += spots.astype(np.int64)
    return f.astype(np.uint16)


@pytest.mark.parametrize("memory", [0, 3, 17])
@pytest.mark.parametrize("dense", [range(0, 4), range(150, 154)])
def test_too_dense_before_the_last_window(ctx, memory, dense):
    # every spot within reach of every other; nothing is left for the windows that follow
    f = grids(300, dense)
    kw = dict(minmass=1000.0, memory=memory, tqdm=False)
    assert list(gt.batch(f[dense[0]:dense[0] + 2], 9, minmass=1000.0, tqdm=False)["frame"]) == [0] * 100 + [1] * 100
    for _ in range(3):
        with pytest.raises(ValueError, match="abnormally high"):
            gt.batch(f, 9, search_range=400.0, **kw)
    assert gt.batch(f, 9, search_range=2.0, **kw)["particle"].max() == 99
