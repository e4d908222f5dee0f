"""The rules by which large tensors are interpolated sheet by sheet (``csrc/interpolate.cu``), asked on the host."""
import ctypes

import pytest

from distdl_b200 import _native

pytestmark = pytest.mark.skipif(not _native.available(), reason="native library not built")
FP32, FP64, BF16 = range(3)


def marches(adjoint, dtype, planes, n_in, n_out, linear=1, corners=0, x_off=None, y_off=None, in_global=None, out_global=None):
    nd = len(n_in)
    ints = lambda a: (ctypes.c_int * nd)(*a)  # noqa: E731
    gi, go, none = in_global or n_in, out_global or n_out, (0,) * nd
    steps = (ctypes.c_double * nd)(*(a / b for a, b in zip(gi, go)))
    return bool(_native.lib().dd_interpolate_marches(linear, adjoint, dtype, nd, ctypes.c_longlong(planes), ints(n_in),
                                                     ints(n_out), ints(x_off or none), ints(y_off or none), ints(gi),
                                                     ints(go), steps, corners))


@pytest.mark.parametrize("dtype,planes,n_in,n_out,want", [
    (BF16, 512, (128, 128), (256, 256), True), (FP32, 72, (64, 64), (128, 128), True),
    (BF16, 147456, (8, 8), (16, 16), False), (BF16, 9216, (32, 32), (64, 64), False),       # short rows: lanes without one
    (BF16, 288, (32, 32), (64, 64), True), (FP32, 288, (32, 32), (64, 64), True),          # ... but few outputs in all
    (FP32, 576, (128, 128), (256, 256), False),                                             # beyond L2
    (BF16, 288, (256, 256), (256, 256), False), (BF16, 576, (256, 256), (128, 128), False),  # no row is read twice
    (FP32, 32, (46, 46, 46), (69, 69, 69), True), (BF16, 288, (34, 34, 34), (68, 68, 68), True),
    (FP32, 18432, (2, 2, 2), (4, 4, 4), False), (BF16, 43691, (4, 4, 4), (6, 6, 6), False),
    (FP32, 2304, (32, 32, 32), (16, 16, 16), False), (FP64, 144, (32, 32, 32), (64, 64, 64), False)])
def test_forward_walks_sheets_only_where_that_is_faster(dtype, planes, n_in, n_out, want):
    assert marches(0, dtype, planes, n_in, n_out) is want


@pytest.mark.parametrize("dtype,planes,n_in,n_out,linear,corners,want", [
    (FP32, 32, (46, 46, 46), (69, 69, 69), 1, 1, True), (BF16, 288, (34, 34, 34), (68, 68, 68), 1, 1, True),
    (FP32, 18432, (2, 2, 2), (4, 4, 4), 1, 0, False), (FP32, 73728, (4, 4, 4), (8, 8, 8), 1, 0, False),   # small sheets
    (FP32, 36, (16, 16, 16), (32, 32, 32), 1, 0, False), (FP32, 128, (16, 16, 16), (32, 32, 32), 1, 0, True),
    (FP32, 128, (16, 16, 16), (32, 32, 32), 0, 0, False),                                    # nearest
    (FP32, 342, (32, 32, 32), (48, 48, 48), 1, 0, False), (FP64, 342, (32, 32, 32), (48, 48, 48), 1, 0, True),
    (FP32, 1152, (32, 32, 32), (32, 32, 32), 1, 0, False), (FP32, 512, (32, 32, 32), (16, 16, 16), 1, 0, True)])
def test_adjoint_walks_sheets_only_where_that_is_faster(dtype, planes, n_in, n_out, linear, corners, want):
    assert marches(1, dtype, planes, n_in, n_out, linear, corners) is want
