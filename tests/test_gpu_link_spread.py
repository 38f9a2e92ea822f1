"""Neighbour search over point sets whose box says little about where the
points are: single points far away, clusters far apart, rows and columns of
one value, coordinates that are not finite.  Ids are the oracle's, and a far
point costs the others nothing."""
import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200 import _ffi
from test_gpu_link_segments import rows

pytestmark = pytest.mark.gpu


def spread(kind, frames=40, n=150, seed=0):
    r = rows(frames, n, 150.0, seed=seed, seen=0.9)
    rng = np.random.default_rng(seed)
    far = rng.random(len(r)) < 0.02
    if kind == "far":
        r[far, 1:] = (rng.uniform(-1, 1, (far.sum(), 2)) * 10.0 ** rng.uniform(2, 12, (far.sum(), 1))).astype(np.float32)
    elif kind == "clusters":        # by the period of the cells and by odd distances
        r[:, 1:] += np.array([[0, 0], [1e5, 0], [0, 4096 * 4.0], [3e6, -7e6]])[rng.integers(0, 4, len(r))]
    elif kind == "line":
        r[:, 1] = 7.0
        r[far, 2] += 1e7
    elif kind == "plane":           # a point a few cells beyond each edge of the repeated ones
        r[:, 1:] *= 30.0
    elif kind == "nonfinite":
        r[far, 1] = rng.choice(np.array([np.nan, np.inf, -np.inf], np.float32), far.sum())
        r[np.roll(far, 5), 2] = rng.choice(np.array([np.nan, np.inf, -np.inf], np.float32), far.sum())
    return r


@pytest.mark.parametrize("memory", [0, 2])
@pytest.mark.parametrize("radius", [0.25, 4.0])
@pytest.mark.parametrize("kind", ["far", "clusters", "line", "plane", "nonfinite"])
def test_ids(oracle, kind, radius, memory):
    if kind == "line" and radius > 1:
        radius = 0.5                # 135 points on 150 pixels
    r = spread(kind)
    assert np.array_equal(gt.link(r, radius, memory), oracle.link(r, radius, memory))


def test_a_far_point_costs_nothing():
    ctx = _ffi.context(0)

    def lists(r):
        gt.link(r, 5.0, 0)
        ctx.profile(True)
        for _ in range(3):
            gt.link(r, 5.0, 0)
        ms = ctx.profile_read("link_lists")[1]
        ctx.profile(False)
        return ms

    rng = np.random.default_rng(0)
    pos = rng.uniform(0, 4096, (10000, 2))
    near = np.concatenate([np.column_stack([np.full(10000, t), pos + rng.normal(0, 0.5, pos.shape)])
                           for t in range(10)]).astype(np.float32)
    far = near.copy()
    far[::10000, 1:] = 1e6
    # with all but one point in a cell: over thirty times
    assert lists(far) < 4 * lists(near)
