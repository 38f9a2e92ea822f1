"""characterize_points over the ways its frames and bandpass take: the strip
kernel (smoothing radius 3-10) and the tile kernel beside it, frames read in
place, frames skipped (a frame without points is not read) and host frames
large enough for the upload lanes."""
import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200._params import trackpy_params
from synth import video

pytestmark = pytest.mark.gpu

COLS = ["y", "x", "mass", "Rg", "raw", "signal", "ecc", "raw_mass", "raw_bg_median", "raw_mass_corrected"]


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("diameter", [5, 7, 21, 23])
@pytest.mark.parametrize("frames", [(0, 1, 2, 3), (1, 4, 5), (2,)])
def test_points_match_detections(oracle, dtype, diameter, frames):
    # points at the places that `batch` finds have the columns it gives them
    f, _ = video(6, 90, 133, n_spots=14, seed=diameter, dtype=dtype, amp_mu=np.log(150.0), bg=60.0, sigma=2.0,
                 read_noise=4.0 if dtype == np.float32 else None)
    tab = oracle.batch(trackpy_params(diameter, minmass=40.0), f.astype(np.float32))
    from gpu_tracking_b200._params import COLUMN_INDEX as ix
    tab = tab[np.isin(tab[:, ix["frame"]], frames)]
    pts = tab[:, [ix["frame"], ix["y"], ix["x"]]].astype(np.float32)
    import torch
    for src in (f, torch.from_numpy(f).cuda()):
        df = gt.characterize_points(src, pts, diameter, has_frames=True, tqdm=False)
        assert np.array_equal(df["frame"].to_numpy(), tab[:, ix["frame"]].astype(np.int64))
        for c in COLS:
            if c in ("mass", "Rg", "ecc"):
                continue   # of the rounded position here, of the walk's last one there
            assert np.array_equal(df[c].to_numpy(np.float32), tab[:, ix[c]].astype(np.float32)), c


def test_points_through_the_upload_lanes():
    import pandas as pd
    import torch
    f, truth = video(40, 400, 301, n_spots=8, seed=4)
    pts = np.concatenate([np.column_stack([np.full(len(t), k), t]) for k, t in enumerate(truth)]).astype(np.float32)
    a = gt.characterize_points(f, pts, 9, has_frames=True, tqdm=False)
    b = gt.characterize_points(torch.from_numpy(f).cuda(), pts, 9, has_frames=True, tqdm=False)
    assert f.nbytes > 4 << 20 and len(a) == len(pts)
    pd.testing.assert_frame_equal(a, b, check_exact=True)
