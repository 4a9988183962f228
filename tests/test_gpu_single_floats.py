"""GPU suite: pixel-major outputs whose rows cannot be stored in float pairs -- an odd kernel count, an output base of 4 bytes -- on
tiles of 256 kernels, single blocks and block pairs."""
import numpy as np
import pytest

import fastertnn_b200 as ft
from cases import BTN, TNN, make_case, threaded_conv, to_nchw, to_nhwc, wgt_ternary
from fastertnn_b200.workloads import Layer

pytestmark = pytest.mark.gpu

# one, two and four taps per stage; kernel counts that end inside a float pair, a slice and a tile; few tiles and several per pair; an even
# count (for the shifted base)
LAYERS = [
    (Layer(192, 23, 23, 257, 1, 1, 0, 1), 40), (Layer(64, 24, 24, 511, 3, 3, 1, 1), 40), (Layer(128, 24, 24, 301, 3, 3, 1, 2), 40),
    (Layer(256, 16, 16, 385, 3, 3, 1, 1), 45), (Layer(256, 12, 12, 256, 3, 3, 1, 1), 30), (Layer(512, 8, 8, 289, 3, 3, 1, 1), 60),
]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("type_", [TNN, BTN])
@pytest.mark.parametrize("layer,N", LAYERS, ids=lambda v: str(v).replace(" ", ""))
def test_single_floats(layer, N, type_, shift, gpu_ctx, checker):
    case = make_case(type_, layer, N, 9500 + layer.KN, "uniform")
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    want = threaded_conv(checker, type_, case.x, case.thr, wp, layer)
    ctx = gpu_ctx
    w = ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    d_x, d_t, d_y = ctx.to_device(to_nhwc(case.x)), ctx.to_device(case.thr), ctx.malloc(want.nbytes + 16)
    try:
        ctx.fill(d_y, np.full(want.size + 4, np.nan, np.float32))
        for _ in range(2):
            ctx.conv(w, d_x, d_t, d_y + 4 * shift, layer.shape(N), case.alpha, ft.NHWC)
        ctx.sync()
        got = ctx.to_host(d_y, (want.size + 4,), np.float32)
        body = got[shift:shift + want.size].reshape(N, layer.OH, layer.OW, layer.KN)
        assert to_nchw(body).tobytes() == want.tobytes()
        assert np.isnan(got[:shift]).all() and np.isnan(got[shift + want.size:]).all()
    finally:
        for p in (d_x, d_t, d_y):
            ctx.free(p)
        w.free()
