"""Child records are read 32 bytes at a time: queries refuse records that are
not 32-byte aligned, before any CUDA call (host pointers here are never read)."""

import ctypes

from atom3d_b200 import _lib
from atom3d_b200.batch import BvhBatch, _bind

ARGUMENT = 1
BUF = 1 << 20  # an aligned address; nothing reads it


def test_single_mesh_queries_refuse_misaligned_records(lib):
    view = _lib.BvhView(BUF, BUF, 1, 1, (ctypes.c_float * 3)(), (ctypes.c_float * 3)())
    for off in (4, 16):
        st = lib.a3d_udf_children(ctypes.byref(view), BUF + off, BUF, 1, BUF, BUF, BUF, None, None, None, None, 1, BUF,
                                  1 << 24, None)
        assert st == ARGUMENT and b"32-B aligned" in lib.a3d_last_error()


def test_batch_queries_refuse_misaligned_records(lib):
    b = BvhBatch(BUF, BUF, 1, 1, BUF, BUF)
    for off in (4, 16):
        st = _bind().a3d_batch_udf_children(ctypes.byref(b), BUF + off, 1, BUF, BUF, 1, BUF, BUF, BUF, None, None, None,
                                            BUF, 1 << 30, None)
        assert st == ARGUMENT and b"32-B aligned" in lib.a3d_last_error()
