"""Tables of a call with a huge radius belong to the call."""
import gc
import os

import numpy as np
import pytest

import gpu_tracking_b200 as gt

pytestmark = pytest.mark.gpu


def resident():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * os.sysconf("SC_PAGE_SIZE")


def points(r):
    return np.array([[60.0, 70.0, r], [31.5, 40.25, 3.0]], np.float32)


def test_large_radius_leaves_no_host_memory():
    f = np.random.default_rng(0).integers(50, 200, (1, 128, 128)).astype(np.uint16)
    small = gt.characterize_points(f, points(5.0), 9, has_r=True, tqdm=False)
    gc.collect()
    before = resident()
    big = gt.characterize_points(f, points(300.0), 9, has_r=True, tqdm=False)   # tables of 290 MB
    assert resident() - before < 100 << 20
    # the tables of the smaller radius are the first part of the larger one's
    assert np.array_equal(small.to_numpy()[1], big.to_numpy()[1], equal_nan=True)
    again = gt.characterize_points(f, points(5.0), 9, has_r=True, tqdm=False)
    assert np.array_equal(small.to_numpy(), again.to_numpy(), equal_nan=True)


@pytest.mark.parametrize("r", [63.0, 64.0, 65.0, 66.0])
def test_radii_about_the_shared_tables(r):
    f = np.random.default_rng(0).integers(50, 200, (1, 160, 160)).astype(np.uint16)
    pts = np.array([[80.0, 80.0, r], [79.5, 81.25, 3.0]], np.float32)
    both = gt.characterize_points(f, pts, 9, has_r=True, tqdm=False)
    alone = gt.characterize_points(f, np.vstack([pts, [[80.0, 80.0, 100.0]]]).astype(np.float32), 9, has_r=True,
                                   tqdm=False)
    assert np.array_equal(both.to_numpy(), alone.to_numpy()[:2], equal_nan=True)
    assert np.isfinite(both["ecc"].to_numpy()).all()
