"""The LoG scale space at the edges of its 34 x 128 tiles and for radii that
take their taps from the kernel parameter (distinct tap counts) or from global
memory (two radii with the same count), up to the largest radius it covers."""
import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200._params import log_params
from synth import video
from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu
COLS = ["frame", "y", "x", "mass", "r"]


@pytest.mark.parametrize("shape", [(2, 33, 127), (1, 34, 128), (1, 35, 129), (2, 68, 40), (1, 103, 261)])
@pytest.mark.parametrize("radii", [dict(lo=2.0, hi=8.0, n=6), dict(lo=2.0, hi=3.0, n=5), dict(lo=1.0, hi=11.0, n=3)])
@pytest.mark.parametrize("dtype", [np.float32, np.uint16])
def test_tiles_match_oracle(oracle, shape, radii, dtype):
    f, _ = video(*shape, n_spots=9, seed=shape[1] + radii["n"], dtype=dtype, sigma_range=(1.4, 4.0), bg=50.0,
                 read_noise=4.0 if dtype == np.float32 else None)
    kw = dict(n_radii=radii["n"], log_spacing=True, minmass=20.0)
    df = gt.LoG(f, radii["lo"], radii["hi"], tqdm=False, **kw)
    assert_same(df, oracle.batch(log_params(radii["lo"], radii["hi"], **kw), f.astype(np.float32)), COLS)
