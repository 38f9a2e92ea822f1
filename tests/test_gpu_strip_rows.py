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


def awkward(kind, shape, seed):
    """Float frames whose sums meet the divisions' and the zero rows' edges."""
    f, _ = video(*shape, n_spots=12, seed=seed, dtype=np.float32, amp_mu=np.log(120.0), bg=60.0, read_noise=4.0)
    rng = np.random.default_rng(seed)
    H, W = shape[1:]
    if kind == "masked":            # zeros, some of them -0, next to data and at every edge
        f[:, : H // 3] = 0.0
        f[:, -H // 4:, : W // 2] = -0.0
        f[:, :, W // 2: W // 2 + 20] = 0.0
    elif kind == "tiny":            # products that underflow, of both signs
        f = (rng.integers(-3, 4, shape) * np.float32(1e-45)).astype(np.float32)
        f[:, H // 2:] *= np.float32(1e20)
    elif kind == "signed":          # sums that cancel to zero
        f = np.where(rng.random(shape) < 0.5, 1.0, -1.0).astype(np.float32)
        f[:, ::2] = -f[:, 1::2][:, : f[:, ::2].shape[1]] if H % 2 == 0 else f[:, ::2]
    elif kind == "huge":            # beyond the proven range of the fast division
        f = f * np.float32(1e30)
    else:                           # NaN and infinities
        f[:, H // 3, W // 3] = np.nan
        f[:, 2, 5] = np.inf
        f[:, -3, -4] = -np.inf
    return f


@pytest.mark.parametrize("kind", ["masked", "tiny", "signed", "huge", "nonfinite"])
@pytest.mark.parametrize("truncate", [True, False])
@pytest.mark.parametrize("diameter,shape", [(9, (2, 70, 150)), (11, (1, 264, 131)), (13, (1, 41, 40))])
def test_float_pixels_at_the_divisions_edges(oracle, kind, truncate, diameter, shape):
    f = awkward(kind, shape, seed=diameter)
    kw = dict(minmass=1e-30, truncate_preprocessed=truncate)
    df = gt.batch(f, diameter, tqdm=False, **kw)
    assert_same(df, oracle.batch(trackpy_params(diameter, **kw), f), ALL_TP)


@pytest.mark.parametrize("kind", ["masked", "tiny"])
def test_log_bandpass_at_the_divisions_edges(oracle, kind):
    from gpu_tracking_b200._params import log_params
    f = awkward(kind, (1, 90, 140), seed=3)
    kw = dict(n_radii=4, minmass=1e-30, overlap_threshold=1.0)
    df = gt.LoG(f, 2.0, 5.0, tqdm=False, **kw)
    assert_same(df, oracle.batch(log_params(2.0, 5.0, **kw), f), ["frame", "y", "x", "mass", "r"])
