"""Seed patches of the learned walk: rows and half columns in registers
(smoothing radius equal to the circle radius or one more) or an output a lane
(other radii), sliding boxcar sums for whole numbers, windows inside the frame
and across its edges.  Rows of integer frames and of the same values in
float32 are equal bit for bit, and so is every row that ends where a walk of
`batch` ends."""
import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200 import learned
from synth import video

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("diameter", [5, 9, 11, 15])
@pytest.mark.parametrize("more", [-2, 0, 2])
@pytest.mark.parametrize("shape,dtype", [((57, 61), np.uint16), ((132, 95), np.uint8)])
def test_seed_patches_against_plain_walks(diameter, more, shape, dtype):
    smoothing = diameter + more
    if smoothing < 3 or smoothing > 15:
        pytest.skip("smoothing radii 1 to 7")
    f, _ = video(3, *shape, 20, seed=diameter + 100 * (more + 2), dtype=dtype, amp_mu=np.log(100.0), bg=30.0)
    net = learned.ProposalNet(seed=0)
    net.threshold = -1e9
    kw = dict(minmass=40.0, smoothing_size=smoothing)
    a = learned.batch_learned(f, diameter, net, **kw)
    b = learned.batch_learned(f.astype(np.float32), diameter, net, **kw)
    assert len(a) > 0 and list(a.columns) == list(b.columns)
    assert np.array_equal(a.to_numpy(), b.to_numpy(), equal_nan=True)
    plain = gt.batch(f, diameter, tqdm=False, **kw)
    at = {r[:3].tobytes(): r for r in np.ascontiguousarray(plain[["frame", "y", "x"] + _values(plain)].to_numpy())}
    same = 0
    for r in np.ascontiguousarray(a[["frame", "y", "x"] + _values(plain)].to_numpy()):
        p = at.get(r[:3].tobytes())
        if p is not None:
            same += 1
            assert np.array_equal(r, p, equal_nan=True)
    assert same > 0


def _values(df):
    return [c for c in df.columns if c not in ("frame", "y", "x", "particle", "duration")]
