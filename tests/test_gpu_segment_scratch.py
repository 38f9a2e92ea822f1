"""Scratch of the linker's segments: bounded whatever edge buffer earlier
calls left behind, and not a reason for a call to fail.  Where it does not fit
the segments get longer, and without any the sequential kernel links; ids and
durations are the oracle's every time."""
import ctypes

import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200._params import trackpy_params
from synth import video
from test_gpu_link_segments import rows
from test_gpu_link_stops import LINK_COLS, ctx, hook  # noqa: F401
from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu

GIB = 1 << 30


@pytest.fixture(scope="module")
def movie():
    return video(150, 64, 64, 14, seed=8, D=1.0, turnover=0.05)[0]


def used():
    import torch
    free, total = torch.cuda.mem_get_info()
    return total - free


def linked(oracle, movie, memory):
    kw = dict(minmass=300.0, search_range=6.0, memory=memory)
    tab = oracle.batch(trackpy_params(9, **kw), movie.astype(np.float32))
    assert_same(gt.batch(movie, 9, tqdm=False, **kw), tab, LINK_COLS)


@pytest.mark.parametrize("edges", [1 << 22, 40 << 20, 400 << 20])
@pytest.mark.parametrize("memory", [0, 3])
def test_bounded_for_large_edge_buffers(oracle, movie, ctx, edges, memory):
    # one run's copy takes 8 bytes an edge: 32 MB, 320 MB (longer segments) and
    # more than all copies together may have (sequential kernel)
    linked(oracle, movie, memory)
    before = used()
    ctx.check(hook("gt__set_link_window_caps", ctypes.c_int64, ctypes.c_int64)(ctx.handle, 0, edges))
    linked(oracle, movie, memory)
    assert used() - before < 8 * edges * 1.2 + 2.3 * GIB


@pytest.mark.parametrize("memory", [0, 2])
def test_sequential_when_there_is_no_memory(oracle, movie, ctx, memory):
    limit = hook("gt__set_optional_limit", ctypes.c_uint64)
    kw = dict(minmass=300.0, search_range=6.0, memory=memory)
    tab = oracle.batch(trackpy_params(9, **kw), movie.astype(np.float32))
    r = rows(300, 300, 250.0, seed=3)
    ids = oracle.link(r, 4.0, memory)
    for bytes_ in (1 << 16, 0):
        ctx.check(limit(ctx.handle, bytes_))
        assert_same(gt.batch(movie, 9, tqdm=False, **kw), tab, LINK_COLS)
        assert np.array_equal(gt.link(r, 4.0, memory), ids)
