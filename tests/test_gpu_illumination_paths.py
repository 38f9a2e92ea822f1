"""Illumination correction and the frame std at the edges of their kernels:
lines of more than one piece and of odd length, smoothing from one tap to far
wider than the frame, frames that do not start on four pixels, sums whose
lengths do not divide by four."""
import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200._params import trackpy_params
from synth import video
from test_gpu_parity import ALL_TP, assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 45, 61), (2, 40, 1100), (5, 1030, 36), (1, 64, 64)])
@pytest.mark.parametrize("sigma", [0.1, 2.0, 30.0, 200.0])
@pytest.mark.parametrize("per_frame,dtype", [(False, np.uint16), (True, np.uint8), (False, np.float32)])
def test_illumination_matches_oracle(oracle, shape, sigma, per_frame, dtype):
    f, _ = video(*shape, n_spots=12, seed=int(sigma) + shape[2], dtype=dtype, amp_mu=np.log(150.0), bg=60.0,
                 read_noise=4.0 if dtype == np.float32 else None)
    kw = dict(minmass=0.5, illumination_sigma=sigma, illumination_correction_per_frame=per_frame)
    df = gt.batch(f, 7, tqdm=False, **kw)
    assert_same(df, oracle.batch(trackpy_params(7, **kw), f.astype(np.float32)), ALL_TP)


@pytest.mark.parametrize("shape", [(2, 8, 8), (2, 16, 32), (3, 64, 24), (2, 128, 96)])
@pytest.mark.parametrize("dtype", [np.uint16, np.uint8, np.float32])
def test_std_matches_oracle(oracle, shape, dtype):
    import torch
    f, _ = video(shape[0] + 1, *shape[1:], n_spots=4, seed=shape[2], dtype=dtype, amp_mu=np.log(150.0), bg=60.0,
                 margin=1.0, read_noise=4.0 if dtype == np.float32 else None)
    kw = dict(snr=0.3, minmass_snr=0.2, adaptive_background=2)
    want = oracle.batch(trackpy_params(5, **kw), f[1:].astype(np.float32))
    assert_same(gt.batch(f[1:], 5, tqdm=False, **kw), want, ALL_TP)
    # the same frames at a device address one pixel off the alignment
    flat = torch.zeros(f[1:].size + 1, dtype=torch.from_numpy(f).dtype, device="cuda")
    flat[1:] = torch.from_numpy(f[1:].reshape(-1)).cuda()
    assert_same(gt.batch(flat[1:].view(f[1:].shape), 5, tqdm=False, **kw), want, ALL_TP)
