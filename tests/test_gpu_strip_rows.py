"""Short strip segments: a grid that would leave SMs idle cuts its frames into
tiles of few rows.  Frames whose heights lie at and next to multiples of the
8-row step, one and several frames a call, every pixel type, equal the oracle."""
import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200._params import trackpy_params
from synth import video
from test_gpu_parity import ALL_TP, assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint16, np.uint8, np.float32])
@pytest.mark.parametrize("shape", [(1, 23, 40), (1, 64, 131), (1, 65, 300), (2, 513, 129), (1, 520, 64), (5, 263, 260)])
@pytest.mark.parametrize("diameter", [5, 11])
def test_short_segments_match_oracle(oracle, dtype, shape, diameter):
    frames, _ = video(*shape, n_spots=max(4, shape[1] * shape[2] // 900), seed=shape[1] + diameter, dtype=dtype,
                      amp_mu=np.log(120.0), bg=60.0, read_noise=4.0 if dtype == np.float32 else None)
    kw = dict(minmass=30.0)
    df = gt.batch(frames, diameter, tqdm=False, **kw)
    tab = oracle.batch(trackpy_params(diameter, **kw), frames.astype(np.float32))
    assert_same(df, tab, ALL_TP)
