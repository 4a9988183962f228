"""GPU suite: layers with few output tiles, which the tensor-copy fed GEMM cuts into narrower kernel tiles than the weight
image's own."""
import numpy as np
import pytest

import fastertnn_b200 as ft
from cases import BNN, BTN, TBN, TNN, make_case, threaded_conv, to_nchw, to_nhwc, wgt_ternary
from fastertnn_b200.workloads import Layer

pytestmark = pytest.mark.gpu

# kernel counts around the tile widths, row counts around the row tile, one stage and many, one, two and four taps per stage,
# and batches on either side of the point where the narrower tiles would no longer fit the chip in one wave (148 SMs)
LAYERS = [
    (Layer(256, 8, 8, 65, 3, 3, 1, 1), 1), (Layer(256, 16, 16, 128, 1, 1, 0, 1), 3), (Layer(64, 9, 14, 129, 3, 3, 1, 2), 2),
    (Layer(128, 14, 14, 191, 3, 3, 1, 2), 5), (Layer(512, 7, 7, 257, 3, 3, 1, 1), 8), (Layer(512, 7, 7, 513, 1, 1, 0, 1), 3),
    (Layer(256, 12, 12, 320, 5, 3, 1, 2), 4), (Layer(1024, 1, 1, 1000, 1, 1, 0, 1), 129), (Layer(256, 16, 16, 256, 1, 1, 0, 1), 18),
    (Layer(256, 16, 16, 256, 1, 1, 0, 1), 19), (Layer(256, 16, 16, 200, 1, 1, 0, 1), 37), (Layer(256, 16, 16, 200, 1, 1, 0, 1), 38),
    # narrow tiles, some blocks with two and more: drained by groups of warps in turn
    (Layer(64, 16, 16, 64, 3, 3, 1, 2), 310), (Layer(256, 16, 16, 100, 1, 1, 0, 1), 150), (Layer(64, 16, 16, 60, 3, 3, 1, 1), 150),
    (Layer(128, 14, 14, 128, 3, 3, 1, 1), 75),
]


@pytest.mark.parametrize("type_", [TNN, TBN, BTN, BNN])
@pytest.mark.parametrize("layer,N", LAYERS, ids=lambda v: str(v).replace(" ", ""))
def test_few_tiles(layer, N, type_, gpu_ctx, checker):
    case = make_case(type_, layer, N, 9100 + layer.KN, "uniform")
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    want = threaded_conv(checker, type_, case.x, case.thr, wp, layer)
    ctx = gpu_ctx
    w = ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    d_t, d_y = ctx.to_device(case.thr), ctx.malloc(want.nbytes)
    try:
        for layout in (ft.NCHW, ft.NHWC):
            d_x = ctx.to_device(case.x if layout == ft.NCHW else to_nhwc(case.x))
            ctx.fill(d_y, np.full(want.size, np.nan, np.float32))
            for _ in range(2):  # the second launch's set-up and weight copies overlap the first launch
                ctx.conv(w, d_x, d_t, d_y, layer.shape(N), case.alpha, layout)
            ctx.sync()
            got = ctx.to_host(d_y, want.shape if layout == ft.NCHW else (N, layer.OH, layer.OW, layer.KN), np.float32)
            got = got if layout == ft.NCHW else to_nchw(got)
            assert got.tobytes() == want.tobytes(), layout
            ctx.free(d_x)
    finally:
        for p in (d_t, d_y):
            ctx.free(p)
        w.free()
