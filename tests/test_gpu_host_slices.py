"""GPU suite: host-buffer layers around the sizes at which the batch is cut into slices."""
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
