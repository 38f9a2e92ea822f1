"""Tables read back into pinned memory: the values of the other way, and no
device memory of its own."""
import ctypes

import numpy as np
import pytest

import gpu_tracking_b200 as gt
from gpu_tracking_b200 import _ffi, api
from gpu_tracking_b200._params import COLUMN_INDEX

pytestmark = pytest.mark.gpu

COLS = ["frame", "y", "x", "mass", "Rg", "raw", "signal", "ecc", "raw_mass", "raw_bg_median", "raw_mass_corrected"]


@pytest.fixture
def table(monkeypatch):
    """Makes a device table of n rows, NaN among them."""
    made = []

    def make(n):
        f = np.random.default_rng(1).integers(0, 250, (1, 256, 256)).astype(np.uint8)
        f[0, 100:200, 100:200] = 0          # patches without signal: 0 / 0
        pts = np.random.default_rng(2).uniform(20, 230, (n, 2)).astype(np.float32)
        with monkeypatch.context() as m:
            m.setattr(api, "_table_to_frame", lambda ctx, handle, params, has_r=None: handle)
            made.append(gt.characterize_points(f, pts, 9, tqdm=False))
        return made[-1]

    yield make
    for h in made:
        _ffi.lib().gt_table_free(h)


def export(handle, n, address, pinned):
    idx = (ctypes.c_int32 * len(COLS))(*[COLUMN_INDEX[c] for c in COLS])
    if pinned:
        return _ffi.lib().gt_table_export_pinned(handle, idx, len(COLS), address)
    dst = (ctypes.c_void_p * len(COLS))(*[address + 8 * n * k for k in range(len(COLS))])
    return _ffi.lib().gt_table_export(handle, idx, len(COLS), dst)


def block(address, n):
    return np.ctypeslib.as_array((ctypes.c_uint8 * (8 * n * len(COLS))).from_address(address))


@pytest.mark.parametrize("n", [1, 31, 2000, 300000])
def test_both_ways_agree(table, n):
    h = table(n)
    pinned = _ffi.lib().gt_host_alloc(8 * n * len(COLS))
    try:
        a = np.zeros(8 * n * len(COLS), np.uint8)
        assert export(h, n, a.ctypes.data, False) == 0
        block(pinned, n)[:] = 1
        assert export(h, n, pinned, True) == 0
        assert np.array_equal(block(pinned, n), a)                  # bit for bit
        assert n == 1 or np.isnan(a.view(np.float64)).any()
        block(pinned, n)[:] = 1
        assert export(h, n, pinned, False) == 0
        assert np.array_equal(block(pinned, n), a)
        b = np.ones_like(a)                                         # pageable memory is as good
        assert export(h, n, b.ctypes.data, True) == 0
        assert np.array_equal(b, a)
    finally:
        _ffi.lib().gt_host_free(pinned)


def test_without_device_memory(table):
    import torch
    small = table(2000)
    n = 1 << 20
    pinned = _ffi.lib().gt_host_alloc(8 * n * len(COLS))
    try:
        assert export(small, 2000, pinned, True) == 0
        h = table(n)
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        hold = torch.empty(free - (48 << 20), dtype=torch.uint8, device="cuda")   # the columns take 92 MB
        assert export(h, n, pinned, True) == 0
        got = block(pinned, n).copy()
        del hold
        torch.cuda.empty_cache()
        want = np.zeros_like(got)
        assert export(h, n, want.ctypes.data, False) == 0
        assert np.array_equal(got, want)
    finally:
        torch.cuda.empty_cache()
        _ffi.lib().gt_host_free(pinned)
