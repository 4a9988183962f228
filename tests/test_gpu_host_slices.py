"""GPU suite: host-buffer layers around the sizes at which the batch is cut into slices."""
import ctypes

import numpy as np
import pytest

from cases import BNN, TNN, make_case, threaded_conv, wgt_ternary
from fastertnn_b200.workloads import Layer

pytestmark = pytest.mark.gpu


# one slice (also of a single image), two, an uneven last one, all eight; batches smaller than the number of slices their bytes ask for
@pytest.mark.parametrize("type_", [TNN, BNN])
@pytest.mark.parametrize("layer,N", [(Layer(64, 16, 16, 40, 3, 3, 1, 2), 1), (Layer(256, 14, 14, 256, 3, 3, 1, 2), 8), (Layer(64, 64, 64, 64, 3, 3, 1, 1), 4),
                                     (Layer(64, 64, 64, 70, 3, 3, 1, 1), 5), (Layer(96, 64, 64, 64, 3, 3, 1, 1), 19), (Layer(64, 200, 200, 64, 1, 1, 0, 1), 3)],
                         ids=lambda v: str(v).replace(" ", ""))
def test_host_slices(layer, N, type_, gpu_ctx, checker):
    case = make_case(type_, layer, N, 9800 + layer.KN, "uniform")
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    want = threaded_conv(checker, type_, case.x, case.thr, wp, layer)
    w = gpu_ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    try:
        for _ in range(2):
            y = np.full(want.shape, np.nan, np.float32)
            gpu_ctx.conv_host(w, case.x.ctypes.data, case.thr.ctypes.data, y.ctypes.data, layer.shape(N), case.alpha)
            assert y.tobytes() == want.tobytes()
    finally:
        w.free()


# page-locked buffers, whose copies do run beside one another: one slice, two, an uneven last one, tapered ends, all eight
@pytest.mark.parametrize("layer,N", [(Layer(256, 14, 14, 256, 3, 3, 1, 2), 8), (Layer(64, 64, 64, 64, 3, 3, 1, 1), 3), (Layer(64, 64, 64, 70, 3, 3, 1, 1), 5),
                                     (Layer(96, 64, 64, 64, 3, 3, 1, 1), 11), (Layer(64, 56, 56, 64, 3, 3, 1, 1), 25)], ids=lambda v: str(v).replace(" ", ""))
def test_host_slices_of_page_locked_buffers(layer, N, gpu_ctx, checker):
    ctx = gpu_ctx
    case = make_case(TNN, layer, N, 9850 + layer.KN, "uniform")
    wp = checker.pack_weights(wgt_ternary(TNN), case.w, case.w_thr)
    want = threaded_conv(checker, TNN, case.x, case.thr, wp, layer)
    w = ctx.upload_weights(TNN, wp, layer.C, layer.KH, layer.KW)
    h_x, h_y = ctx.malloc_host(case.x.nbytes), ctx.malloc_host(want.nbytes)
    try:
        x, y = (np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_float)), shape=a.shape) for p, a in ((h_x, case.x), (h_y, want)))
        x[:] = case.x
        for _ in range(2):
            y.fill(np.nan)
            ctx.conv_host(w, h_x, case.thr.ctypes.data, h_y, layer.shape(N), case.alpha)
            assert y.tobytes() == want.tobytes()
    finally:
        ctx.free_host(h_x)
        ctx.free_host(h_y)
        w.free()
