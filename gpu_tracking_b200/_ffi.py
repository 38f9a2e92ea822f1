"""ctypes binding of libgt_b200.so (the C ABI of include/gpu_tracking_b200.h).

The library is built in-tree by ``gpu_tracking_b200.build``.  There is no
fallback: if the CUDA library cannot be loaded or no CUDA device is present,
every call raises.
"""
import ctypes
import os
import threading

import numpy as np

from ._params import GtParams

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(HERE, "libgt_b200.so")

GT_OK = 0
STATUS_NAMES = {
    1: "InvalidArgument", 2: "DimensionMismatch", 3: "EmptyIterator", 4: "NonSortedCharacterization",
    5: "FrameOutOfBounds", 6: "NonStandardArrayLayout", 7: "ArrayDimensionsError", 8: "TooDenseToLink",
    9: "Interrupted", 10: "CapacityExceeded", 11: "CudaError", 12: "NoDevice", 13: "SubnetTooExpensive",
    14: "Internal", 15: "FileNotFound", 16: "ReadError",
}

_lib = None
_lock = threading.Lock()


class GpuTrackingError(RuntimeError):
    """Raised for CUDA or internal failures of the engine."""

    def __init__(self, status, message):
        super().__init__("%s: %s" % (STATUS_NAMES.get(status, status), message))
        self.status = status


def to_exception(status, message):
    """Map a gt_status to the exception the reference raises
    (gpu_tracking_python/src/python_bindings.rs:160-193)."""
    if status == 9:
        return KeyboardInterrupt(message)
    if status == 12:
        return ConnectionError(message)
    if status == 15:
        return FileNotFoundError(message)
    if status == 16:
        return ValueError(message)
    if status in (1, 2, 3, 4, 5, 6, 7, 8, 10):
        return ValueError(message)
    return GpuTrackingError(status, message)


class TrainOpts(ctypes.Structure):
    """gt_train_opts (include/gpu_tracking_b200.h)."""
    _fields_ = [("steps", ctypes.c_int32), ("batch", ctypes.c_int32), ("crop", ctypes.c_int32),
                ("lr", ctypes.c_float), ("pos_weight", ctypes.c_float), ("offset_weight", ctypes.c_float),
                ("seed", ctypes.c_uint32)]


def lib():
    global _lib
    with _lock:
        if _lib is not None:
            return _lib
        if not os.path.exists(LIB_PATH):
            from . import build
            build.build()
        L = ctypes.CDLL(LIB_PATH)
        vp, i32, i64, f32 = ctypes.c_void_p, ctypes.c_int32, ctypes.c_int64, ctypes.c_float
        P = ctypes.POINTER
        L.gt_version.restype = ctypes.c_char_p
        L.gt_params_default.argtypes = [P(GtParams)]
        L.gt_create.argtypes = [i32, P(vp)]
        L.gt_destroy.argtypes = [vp]
        L.gt_last_error.argtypes = [vp]
        L.gt_last_error.restype = ctypes.c_char_p
        L.gt_set_interrupt.argtypes = [vp, P(i32)]
        L.gt_progress.argtypes = [vp, P(i64), P(i64)]
        L.gt_table_nrows.argtypes = [vp]
        L.gt_table_nrows.restype = i64
        L.gt_table_column_f32.argtypes = [vp, i32, P(f32)]
        L.gt_table_column_i64.argtypes = [vp, i32, P(i64)]
        L.gt_table_export.argtypes = [vp, P(i32), i32, P(vp)]
        L.gt_table_export_pinned.argtypes = [vp, P(i32), i32, vp]
        L.gt_host_alloc.argtypes = [ctypes.c_size_t]
        L.gt_host_alloc.restype = vp
        L.gt_host_free.argtypes = [vp]
        L.gt_table_has_column.argtypes = [vp, i32]
        L.gt_table_has_column.restype = i32
        L.gt_table_free.argtypes = [vp]
        L.gt_batch.argtypes = [vp, P(GtParams), vp, i32, i64, i32, i32, P(i64), P(i64), i64, P(vp)]
        L.gt_batch_videos.argtypes = [vp, P(GtParams), i32, P(vp), i32, P(i64), P(i32), P(i32), P(vp)]
        L.gt_characterize_points.argtypes = [vp, P(GtParams), vp, i32, i64, i32, i32, P(f32), i64, i32, i32,
                                             P(vp)]
        L.gt_link.argtypes = [vp, P(f32), i64, f32, ctypes.c_uint32, P(i64)]
        L.gt_connect.argtypes = [vp, P(f32), i64, P(f32), i64, f32, P(i64), P(i64)]
        L.gt_mean_frame.argtypes = [vp, vp, i32, i64, i32, i32, P(f32)]
        L.gt_profile_enable.argtypes = [vp, i32]
        L.gt_profile_read.argtypes = [vp, ctypes.c_char_p, P(i64), P(ctypes.c_double)]
        L.gt_launch_count.argtypes = [vp]
        L.gt_launch_count.restype = i64
        L.gt_train_opts_default.argtypes = [P(TrainOpts)]
        L.gt_proposal_num_params.restype = i64
        L.gt_proposal_create.argtypes = [vp, ctypes.c_uint64, P(vp)]
        L.gt_proposal_destroy.argtypes = [vp]
        L.gt_proposal_set.argtypes = [vp, vp, P(f32), f32, f32, f32]
        L.gt_proposal_get.argtypes = [vp, vp, P(f32), P(f32), P(f32), P(f32)]
        L.gt_proposal_train.argtypes = [vp, vp, vp, i32, i64, i32, i32, P(i64), P(f32), P(f32), i64, P(TrainOpts),
                                        P(f32)]
        L.gt_proposal_maps.argtypes = [vp, vp, vp, i32, i64, i32, i32, P(f32)]
        L.gt_batch_learned.argtypes = [vp, P(GtParams), vp, vp, i32, i64, i32, i32, P(i64), P(i64), i64, P(vp)]
        L.gt_video_open.argtypes = [ctypes.c_char_p, i32, P(vp)]
        L.gt_video_open.restype = i32
        L.gt_video_info.argtypes = [vp, P(i64), P(i32), P(i32), P(i32)]
        L.gt_video_info.restype = i32
        L.gt_video_read.argtypes = [vp, P(i64), i64, i32, vp]
        L.gt_video_read.restype = i32
        L.gt_video_read_device.argtypes = [vp, vp, P(i64), i64, i32, vp]
        L.gt_video_read_device.restype = i32
        L.gt_video_close.argtypes = [vp]
        L.gt_video_last_error.restype = ctypes.c_char_p
        L.gt_last_walk_starts.argtypes = [vp]
        L.gt_last_walk_starts.restype = i64
        L.gt__proposal_loss_grad.argtypes = [vp, vp, vp, i32, i64, i32, i32, P(i64), P(f32), P(f32), i64, P(i32), i32,
                                             i32, f32, f32, P(f32), P(f32)]
        for name in ("gt_create", "gt_set_interrupt", "gt_progress", "gt_table_column_f32", "gt_table_column_i64",
                     "gt_table_export", "gt_table_export_pinned", "gt_batch", "gt_batch_videos", "gt_characterize_points", "gt_link", "gt_connect", "gt_mean_frame",
                     "gt_profile_enable", "gt_profile_read", "gt_proposal_create", "gt_proposal_set",
                     "gt_proposal_get", "gt_proposal_train", "gt_proposal_maps", "gt_batch_learned",
                     "gt__proposal_loss_grad"):
            getattr(L, name).restype = i32
        _lib = L
        return L


class Context:
    """One engine context (device, streams, persistent device buffers)."""

    def __init__(self, device=0):
        self._h = ctypes.c_void_p()
        st = lib().gt_create(int(device), ctypes.byref(self._h))
        if st != GT_OK:
            raise to_exception(st, "could not create a context on CUDA device %d" % device)
        self.device = device
        self._flag = ctypes.c_int32(0)
        lib().gt_set_interrupt(self._h, ctypes.byref(self._flag))

    @property
    def handle(self):
        return self._h

    def check(self, st):
        if st != GT_OK:
            msg = lib().gt_last_error(self._h)
            raise to_exception(st, msg.decode() if msg else "")

    def interrupt(self, on=True):
        self._flag.value = 1 if on else 0

    def progress(self):
        d, t = ctypes.c_int64(), ctypes.c_int64()
        lib().gt_progress(self._h, ctypes.byref(d), ctypes.byref(t))
        return d.value, t.value

    def profile(self, enable=True):
        self.check(lib().gt_profile_enable(self._h, 1 if enable else 0))

    def profile_read(self, name):
        n, ms = ctypes.c_int64(), ctypes.c_double()
        self.check(lib().gt_profile_read(self._h, name.encode(), ctypes.byref(n), ctypes.byref(ms)))
        return n.value, ms.value

    def launch_count(self):
        return lib().gt_launch_count(self._h)

    def close(self):
        if self._h:
            lib().gt_destroy(self._h)
            self._h = ctypes.c_void_p()
            results.trim()

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


class _Block:
    """Host memory of one result column.  The arrays made from it keep it alive;
    when the last of them goes, its memory goes back to the pool."""

    def __init__(self, pool, size, address, keep=None, slab=None):
        self._pool, self._size, self._address, self._keep, self._slab = pool, size, address, keep, slab
        self.__array_interface__ = {"shape": (size,), "typestr": "|u1", "data": (address, False), "version": 3}

    @property
    def address(self):
        return self._address

    @property
    def pinned(self):
        return self._keep is None

    def __del__(self):
        try:
            self._pool._back(self)
        except Exception:
            pass


class _Slab:
    """Blocks that were pinned together; `out` of them are in results."""

    def __init__(self, address, size, parts):
        self.address, self.size, self.parts, self.out = address, size, parts, parts


class ResultPool:
    """Host memory for the columns of large results.

    Every column has a block of its own (an eighth larger than the column at
    most), so a column that is kept keeps nothing else.  The memory of a
    dropped column serves the next one of its size (88 MB of columns: 5.6-7.6
    ms into fresh memory, which faults page by page, 2.9-3.8 ms into memory
    used before).  Pinned memory the device fills by itself (1.7 ms; 26 MB 0.5
    instead of 1.4-1.9, 3.5 MB 0.09 instead of 0.25), but pinning takes about
    0.4 ms a megabyte and 2.4 ms at least: what 12 to 20 tables save up to 32
    MB and 30 to 36 above.  So the columns of a table are pinned, all at once,
    when `earned` tables of their size were dropped: a program that keeps its
    tables, or makes few, does not pay for it.  Tables above a quarter of
    `limit` are never pinned.  At most `limit` bytes are pinned, in use and
    idle together, and at most as many idle bytes of ordinary memory are kept.
    """

    PIN_AFTER = 18

    def earned(self, size):
        return self.PIN_AFTER if size <= 4 << 20 else 2 * self.PIN_AFTER

    def __init__(self, limit=512 << 20):
        self._lock = threading.RLock()   # a block may go while another is taken
        self._limit, self._pinned, self._kept = limit, 0, 0
        self._idle, self._ordinary, self._dropped = {}, {}, {}

    @staticmethod
    def block_size(nbytes):
        """The size of the block for nbytes: eight sizes to a power of two, at least 64 KB."""
        top = 1 << max(16, (max(int(nbytes), 1) - 1).bit_length())
        step = top // 16 if top > 1 << 16 else top
        return -(-max(int(nbytes), 1) // step) * step

    def take(self, nbytes):
        return self.take_columns(nbytes, 1)[0]

    def take_columns(self, nbytes, count):
        """`count` blocks of nbytes, pinned all of them or none."""
        size = self.block_size(nbytes)
        kept = []
        with self._lock:
            idle = self._idle.get(size, [])
            if len(idle) >= count:
                return [self._out(size, *idle.pop()) for _ in range(count)]
            ordinary = self._ordinary.get(size, [])
            need = self.earned(size) * count
            pin = (self._dropped.get(size, 0) >= need and size * count <= self._limit // 4
                   and self._pinned + size * count <= self._limit)
            if pin:
                self._dropped[size] -= need
                self._pinned += size * count
            else:
                kept = [ordinary.pop() for _ in range(min(count, len(ordinary)))]
                self._kept -= size * len(kept)
        if pin:
            address = lib().gt_host_alloc(size * count)
            if address:
                slab = _Slab(address, size, count)
                return [_Block(self, size, address + size * k, slab=slab) for k in range(count)]
            with self._lock:
                self._pinned -= size * count
        kept += [np.empty(size, np.uint8) for _ in range(count - len(kept))]
        return [_Block(self, size, a.ctypes.data, a) for a in kept]

    def _out(self, size, address, slab):
        slab.out += 1
        return _Block(self, size, address, slab=slab)

    def _back(self, block):
        size = block._size
        with self._lock:
            if block.pinned:
                block._slab.out -= 1
                self._idle.setdefault(size, []).append((block._address, block._slab))
                return
            # as many as a table of every column pins, twice
            self._dropped[size] = min(2 * 32 * self.earned(size), self._dropped.get(size, 0) + 1)
            if self._kept + size <= self._limit:
                self._ordinary.setdefault(size, []).append(block._keep)
                self._kept += size

    def trim(self):
        """Gives the idle memory back to the system (pinned blocks when all
        that were pinned with them are idle)."""
        free = {}
        with self._lock:
            self._ordinary, self._kept = {}, 0
            for size, idle in self._idle.items():
                free.update((slab.address, slab) for _, slab in idle if not slab.out)
                self._idle[size] = [part for part in idle if part[1].out]
            for slab in free.values():
                self._pinned -= slab.size * slab.parts
        for address in free:
            lib().gt_host_free(address)


results = ResultPool()
_contexts = {}


def context(device=0):
    """The process-wide context of a device (created on first use)."""
    with _lock:
        ctx = _contexts.get(device)
    if ctx is None:
        ctx = Context(device)
        with _lock:
            _contexts[device] = ctx
    return ctx
