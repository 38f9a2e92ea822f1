"""The linker's frame loop cut into segments that run side by side.

Segments of memory + 2 frames and more start from an empty state a
few frames early; boundaries whose states do not agree are linked again.  Ids
must equal the oracle's whole-video linker whatever the number of frames
(below, at and above whole segments), the memory, the crowding (dense sets,
where most boundaries do not hold) and frames without points, in one video
and in several at once.
"""
import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200._params import trackpy_params
from synth import video
from test_gpu_parity import ALL_TP, assert_same

pytestmark = pytest.mark.gpu


def rows(frames, n, side, seed, seen=0.8, D=1.0, empty=()):
    """(frame, y, x) of n diffusing points, each there with probability `seen`."""
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0, side, (n, 2))
    out = []
    for t in range(frames):
        pos = np.clip(pos + rng.normal(0, np.sqrt(2 * D), pos.shape), 0, side)
        there = rng.random(n) < (0.0 if t in empty else seen)
        out.append(np.column_stack([np.full(there.sum(), t), pos[there]]))
    return np.concatenate(out).astype(np.float32)


@pytest.mark.parametrize("memory", [0, 1, 3, 5])
@pytest.mark.parametrize("frames", [2, 3, 4, 5, 6, 7, 8, 9, 15, 16, 17, 31, 100])
def test_link_over_segment_edges(oracle, memory, frames):
    r = rows(frames, 60, 120.0, seed=frames + 10 * memory)
    assert np.array_equal(gt.link(r, 4.0, memory), oracle.link(r, 4.0, memory))


@pytest.mark.parametrize("memory", [0, 1, 2, 4])
@pytest.mark.parametrize("side,radius", [(60.0, 5.0), (45.0, 4.0)])
def test_link_crowded(oracle, memory, side, radius):
    # many shared neighbours: what old ring entries took changes the boundaries
    r = rows(120, 40, side, seed=int(side) + memory, seen=0.6, D=2.0)
    assert np.array_equal(gt.link(r, radius, memory), oracle.link(r, radius, memory))


@pytest.mark.parametrize("memory", [0, 2])
def test_link_with_empty_frames(oracle, memory):
    r = rows(70, 30, 90.0, seed=5, empty=(0, 1, 15, 16, 17, 18, 19, 20, 40, 69))
    assert np.array_equal(gt.link(r, 4.0, memory), oracle.link(r, 4.0, memory))


@pytest.mark.parametrize("frames", [130, 145, 260])
@pytest.mark.parametrize("memory", [0, 2, 17])
def test_batch_windows_of_segments(oracle, frames, memory):
    f, _ = video(frames, 64, 64, 14, seed=31 + frames, D=1.0, turnover=0.05)
    kw = dict(minmass=300.0, search_range=6.0, memory=memory)
    df = gt.batch(f, 9, tqdm=False, **kw)
    tab = oracle.batch(trackpy_params(9, **kw), f.astype(np.float32))
    assert_same(df, tab, ALL_TP + ["particle", "duration"])


def test_videos_of_segments(oracle):
    vids = [video(t, 64, 64, 12, seed=40 + t, D=1.0, turnover=0.05)[0] for t in (5, 20, 47, 90)]
    kw = dict(minmass=300.0, search_range=6.0, memory=3)
    for df, f in zip(gt.batch_videos(vids, 9, **kw), vids):
        assert_same(df, oracle.batch(trackpy_params(9, **kw), f.astype(np.float32)), ALL_TP + ["particle", "duration"])
