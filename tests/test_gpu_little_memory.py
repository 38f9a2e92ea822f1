"""Calls on a device with little memory left filter fewer frames a launch."""
import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200 import _ffi

pytestmark = pytest.mark.gpu

FREE = 1600 << 20     # the processed images of 128 frames of 2048^2 take 2 GiB


@pytest.fixture
def frames(monkeypatch):
    """128 frames on the device, a context without buffers, and little memory."""
    import torch
    rng = np.random.default_rng(0)
    one = rng.poisson(40.0, (2048, 2048)).astype(np.uint8)
    for y, x in rng.integers(20, 2028, (150, 2)):
        one[y - 2:y + 3, x - 2:x + 3] += 60
    f = torch.from_numpy(one).cuda().repeat(128, 1, 1)
    for t in range(128):
        f[t] = torch.roll(f[t], t, 1)
    c = _ffi.Context(0)
    monkeypatch.setitem(_ffi._contexts, 0, c)
    gt.batch(f[:2], 9, minmass=500.0, tqdm=False)        # modules and pools of a small call
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - FREE, dtype=torch.uint8, device="cuda")

    def release():
        nonlocal hold
        hold = None
        torch.cuda.empty_cache()

    yield f, release
    release()
    c.close()


def test_batch(frames):
    f, release = frames
    little = gt.batch(f, 9, minmass=500.0, tqdm=False)
    assert len(little) > 5000
    release()
    assert np.array_equal(little.to_numpy(), gt.batch(f, 9, minmass=500.0, tqdm=False).to_numpy(), equal_nan=True)


def test_characterize_points(frames):
    f, release = frames
    pts = np.array([[t, 100.0 + t, 200.0 + 3 * t] for t in range(128)], np.float32)
    little = gt.characterize_points(f, pts, 9, has_frames=True, tqdm=False)
    release()
    assert np.array_equal(little.to_numpy(), gt.characterize_points(f, pts, 9, has_frames=True, tqdm=False).to_numpy(),
                          equal_nan=True)
