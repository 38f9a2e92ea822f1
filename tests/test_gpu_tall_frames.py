"""Frames of more rows than 128 strip segments of 512 rows hold (line scans):
every call that filters with the strip kernel equals the oracle there."""
import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200._params import COLUMN_INDEX, log_params, trackpy_params
from synth import video
from test_gpu_parity import ALL_TP, assert_same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[65536, 65537, 70000])
def tall(request):
    return video(1, request.param, 40, n_spots=400, seed=request.param)[0]


def test_batch(oracle, tall):
    kw = dict(minmass=300.0)
    tab = oracle.batch(trackpy_params(9, **kw), tall.astype(np.float32))
    assert len(tab) > 100
    assert_same(gt.batch(tall, 9, tqdm=False, **kw), tab, ALL_TP)


def test_log(oracle, tall):
    kw = dict(n_radii=3, minmass=400.0)
    tab = oracle.batch(log_params(2.0, 4.0, **kw), tall.astype(np.float32))
    assert_same(gt.LoG(tall, 2.0, 4.0, tqdm=False, **kw), tab, ["frame", "y", "x", "mass", "r"])


def test_characterize_points(oracle, tall):
    tab = oracle.batch(trackpy_params(9, minmass=300.0), tall.astype(np.float32))
    ix = COLUMN_INDEX
    pts = tab[:, [ix["frame"], ix["y"], ix["x"]]].astype(np.float32)
    df = gt.characterize_points(tall, pts, 9, has_frames=True, tqdm=False)
    for c in ("y", "x", "raw", "signal", "raw_mass", "raw_bg_median", "raw_mass_corrected"):
        assert np.array_equal(df[c].to_numpy(np.float32), tab[:, ix[c]].astype(np.float32)), c
