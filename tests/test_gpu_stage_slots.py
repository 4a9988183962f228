"""GPU suite: rings whose slots hold several stages -- the tensor-copy fed GEMM's pairs of stages on tiles of 64 and 128 kernels and
the slab-fed GEMM's filter rows of 3x3 layers whose weights stream."""
import numpy as np
import pytest

import fastertnn_b200 as ft
from cases import BTN, TNN, make_case, threaded_conv, to_nchw, to_nhwc, wgt_ternary
from fastertnn_b200.api import GEMM_F4_SLAB, GEMM_F4_TC
from fastertnn_b200.workloads import Layer

pytestmark = pytest.mark.gpu

# one stage (half a slot), odd and even numbers of stages, fewer and more than the ring holds, slots that end inside a filter (one, two
# and four taps per stage), several tiles per block, kernel counts around the tiles, one and several channel groups per slab
LAYERS = [
    (Layer(64, 12, 12, 40, 1, 1, 0, 1), 3), (Layer(64, 12, 12, 64, 3, 3, 1, 1), 2), (Layer(64, 16, 16, 64, 5, 5, 2, 2), 90),
    (Layer(128, 12, 12, 100, 3, 3, 1, 2), 3), (Layer(128, 16, 16, 128, 5, 3, 1, 1), 70), (Layer(256, 10, 14, 64, 3, 3, 1, 1), 2),
    (Layer(256, 16, 16, 129, 3, 3, 1, 1), 3), (Layer(256, 20, 20, 100, 3, 3, 1, 1), 60), (Layer(512, 8, 8, 200, 3, 3, 1, 1), 3),
    (Layer(768, 7, 9, 65, 3, 3, 0, 1), 2), (Layer(512, 9, 9, 520, 3, 3, 1, 1), 5), (Layer(1024, 6, 6, 70, 3, 3, 1, 1), 4),
    (Layer(256, 9, 9, 70, 5, 5, 2, 1), 2), (Layer(256, 6, 110, 256, 3, 3, 1, 1), 2),
]


@pytest.mark.parametrize("type_,algo", [(TNN, GEMM_F4_TC), (TNN, GEMM_F4_SLAB), (BTN, GEMM_F4_SLAB)], ids=["im2col", "slab", "slab-btn"])
@pytest.mark.parametrize("layer,N", LAYERS, ids=lambda v: str(v).replace(" ", ""))
def test_stage_slots(layer, N, type_, algo, gpu_ctx, checker):
    if algo == GEMM_F4_SLAB and layer.S != 1:
        pytest.skip("the slab-fed form is for stride-1 layers")
    case = make_case(type_, layer, N, 9700 + layer.KN, "uniform")
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
                ctx.conv(w, d_x, d_t, d_y, layer.shape(N), case.alpha, layout, gemm_algo=algo)
            ctx.sync()
            got = ctx.to_host(d_y, want.shape if layout == ft.NCHW else (N, layer.OH, layer.OW, layer.KN), np.float32)
            got = got if layout == ft.NCHW else to_nchw(got)
            assert got.tobytes() == want.tobytes(), layout
            ctx.free(d_x)
    finally:
        for p in (d_t, d_y):
            ctx.free(p)
        w.free()
