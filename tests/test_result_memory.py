"""A result column holds its own memory and little more, whatever becomes of
the table that it came with; pinned columns are pinned and given back
together."""
import gc

import numpy as np
import pytest

from gpu_tracking_b200 import _ffi, api
from test_result_pool import fake  # noqa: F401


def owner_bytes(a):
    """Bytes of the memory that an array keeps alive."""
    while isinstance(a, np.ndarray) and a.base is not None:
        a = a.base
    return a._size if isinstance(a, _ffi._Block) else a.nbytes


@pytest.mark.parametrize("rows", [0, 1, 1000, 10082, 10083, 1 << 17, 100001, 1 << 20])
def test_columns_own_their_memory(rows):
    cols = api._columns(rows, 13)
    assert len(cols) == 13
    for a in cols:
        assert a.shape == (rows,) and a.dtype == np.int64 and a.flags.writeable and a.flags.c_contiguous
        assert owner_bytes(a) <= max(8 * rows * 1.125, 8 * rows if 8 * rows * 13 <= 1 << 20 else 1 << 16)
    spans = sorted((a.ctypes.data, a.nbytes) for a in cols if rows)
    assert all(p + n <= q for (p, n), (q, _) in zip(spans, spans[1:]))


@pytest.mark.parametrize("nbytes", [1, 65536, 65537, 1 << 17, (1 << 17) + 1, 1 << 20, (1 << 20) + 1, 3 << 20, 12345678])
def test_block_sizes(nbytes):
    size = _ffi.ResultPool.block_size(nbytes)
    assert nbytes <= size <= max(65536, nbytes * 1.125)
    assert _ffi.ResultPool.block_size(size) == size


def test_pinned_columns_come_and_go_together(fake):  # noqa: F811
    pool = _ffi.ResultPool(limit=64 << 20)
    pool.PIN_AFTER = 2
    n = 1 << 20
    for k in range(2):
        held = pool.take_columns(n, 5)
        assert not any(b.pinned for b in held) and not fake.live
        del held
        gc.collect()
    held = pool.take_columns(n, 5)
    assert all(b.pinned for b in held) and len(fake.live) == 1 and pool._pinned == 5 * n
    first = held.pop(0)
    del held
    gc.collect()
    pool.trim()                     # one of them is still in a result
    assert len(fake.live) == 1 and pool._pinned == 5 * n
    four = pool.take_columns(n, 4)
    assert all(b.pinned for b in four) and first.address not in {b.address for b in four}
    assert not pool.take_columns(n, 5)[0].pinned        # not all of them: none
    del four, first
    gc.collect()
    pool.trim()
    assert not fake.live and pool._pinned == 0


def test_pin_failure_gives_ordinary_memory(fake, monkeypatch):  # noqa: F811
    monkeypatch.setattr(fake, "gt_host_alloc", lambda size: None)
    pool = _ffi.ResultPool(limit=64 << 20)
    pool.PIN_AFTER = 1
    for _ in range(4):
        held = pool.take_columns(1 << 20, 3)
        assert len(held) == 3 and not any(b.pinned for b in held) and pool._pinned == 0
        del held
        gc.collect()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [700, 50000])
def test_kept_column_of_a_table(n):
    import gpu_tracking_b200 as gt
    f = np.random.default_rng(1).integers(0, 250, (1, 200, 200)).astype(np.uint8)
    pts = np.random.default_rng(2).uniform(20, 180, (n, 2)).astype(np.float32)
    want = gt.characterize_points(f, pts, 9, tqdm=False).copy(deep=True)
    for k in range(3 * _ffi.results.PIN_AFTER):      # pinned on the way where the table is a large one
        df = gt.characterize_points(f, pts, 9, tqdm=False)
        if k % 8 == 0:
            assert np.array_equal(df.to_numpy(), want.to_numpy(), equal_nan=True)
    for name in ("frame", "y", "mass"):
        a = df[name].to_numpy()
        assert owner_bytes(a) <= max(8 * n * 1.125, 1 << 16)
    kept = df["y"]
    del df
    for _ in range(3):
        gt.characterize_points(f, pts[::-1], 9, tqdm=False)
    assert np.array_equal(kept.to_numpy(), want["y"].to_numpy())
