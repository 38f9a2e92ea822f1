"""Canonical order, filter_close and prune where their counting sorts and
rounds have edges: a row of spots that overfills a bin of candidate pixels
(bitonic order instead), close pairs of equal mass (ties by canonical order),
frames at the largest number of detections that stays in shared memory and
beyond it, blobs that overlap more others than a list holds."""
import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200._params import log_params, trackpy_params
from test_gpu_parity import ALL_TP, assert_same

pytestmark = pytest.mark.gpu


def spots(H, W, at, amp=400, bg=20):
    f = np.full((1, H, W), bg, np.float64)
    yy, xx = np.mgrid[-6:7, -6:7]
    for k, (y, x) in enumerate(at):
        f[0, y - 6:y + 7, x - 6:x + 7] += amp * np.exp(-(yy ** 2 + xx ** 2) / (2 * 1.5 ** 2))
    return f.astype(np.uint16)


def check(oracle, f, d, **kw):
    df = gt.batch(f, d, tqdm=False, **kw)
    assert_same(df, oracle.batch(trackpy_params(d, **kw), f.astype(np.float32)), ALL_TP)
    return df


def test_crowded_bin(oracle):
    # 1600 x 1600: a bin holds 625 pixels, the row a spot every 15
    df = check(oracle, spots(1600, 1600, [(y, x) for y in (300, 301) for x in range(20 + 7 * (y - 300), 1580, 15)]), 7,
               minmass=100.0)
    assert len(df) > 50


@pytest.mark.parametrize("gap", [9, 10, 11])
def test_equal_neighbours(oracle, gap):
    # noiseless pairs: equal masses, the earlier one in canonical order stays
    at = [(y, x + dx) for y in range(20, 180, 30) for x in range(20, 160, 40) for dx in (0, gap)]
    check(oracle, spots(200, 200, at), 9, minmass=50.0, separation=10)


@pytest.mark.parametrize("side", [380, 460, 640])
def test_many_detections(oracle, side):
    rng = np.random.default_rng(side)
    f = rng.poisson(200, (1, side, side)).astype(np.uint16)
    df = check(oracle, f, 5, minmass=0.5, separation=4)
    assert len(df) > side * side // 80


@pytest.mark.parametrize("side,radii", [(64, (2.0, 4.0)), (96, (2.0, 9.0)), (200, (1.5, 6.0))])
@pytest.mark.parametrize("overlap", [0.0, 0.4])
def test_prune_on_noise(oracle, side, radii, overlap):
    rng = np.random.default_rng(side)
    f = rng.normal(50.0, 8.0, (2, side, side)).astype(np.float32)
    kw = dict(n_radii=6, minmass=5.0, overlap_threshold=overlap)
    df = gt.LoG(f, radii[0], radii[1], tqdm=False, **kw)
    assert_same(df, oracle.batch(log_params(radii[0], radii[1], **kw), f), ["frame", "y", "x", "mass", "r"])
