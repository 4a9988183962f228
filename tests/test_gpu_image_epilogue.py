"""GPU suite: the 4-bit image the GEMMs write for a following layer, value by value what quantising their fp32 output gives -- for
every kind of threshold (the epilogue turns PReLU and rule into thresholds on the accumulator), slabs that the loaders fetch and
rings that several tiles of a block pass through."""
import numpy as np
import pytest

import fastertnn_b200 as ft
from cases import BNN, BTN, TBN, TNN, make_case, wgt_ternary
from fastertnn_b200 import api
from fastertnn_b200.workloads import Layer

pytestmark = pytest.mark.gpu

# 32-, 64- and 128-byte pixels; one tile per block, a few, more than the rings hold; whole slices of kernels, a ragged last one, none
# whole; slabs that run past the image's end
LAYERS = [
    (Layer(64, 8, 8, 64, 3, 3, 1, 1), 11), (Layer(64, 32, 32, 64, 3, 3, 1, 1), 70), (Layer(40, 56, 56, 64, 3, 3, 1, 1), 80),
    (Layer(64, 12, 12, 96, 3, 3, 1, 1), 40), (Layer(64, 12, 12, 20, 5, 5, 2, 1), 12), (Layer(128, 8, 12, 128, 3, 3, 1, 1), 30),
    (Layer(128, 28, 28, 128, 3, 3, 1, 1), 70), (Layer(128, 16, 16, 64, 3, 3, 1, 1), 60), (Layer(128, 12, 12, 256, 3, 3, 1, 1), 13),
    (Layer(256, 12, 12, 200, 3, 3, 1, 1), 12), (Layer(512, 8, 8, 130, 3, 3, 1, 1), 15), (Layer(64, 12, 12, 300, 1, 1, 0, 1), 22),
]
THRESHOLDS = np.array([0.25, -0.0, 0.0, -3.0, 5.5, 1e30, -1e30, np.inf, -np.inf, np.nan, 1.0], np.float32)


@pytest.mark.parametrize("type_", [TNN, TBN, BTN, BNN])
@pytest.mark.parametrize("alpha", [0.5, 0.3, 1.0])
@pytest.mark.parametrize("layer,N", LAYERS, ids=lambda v: str(v).replace(" ", ""))
def test_image_epilogue(layer, N, type_, alpha, gpu_ctx, checker):
    ternary = type_ in (TNN, TBN)
    case = make_case(type_, layer, N, 9900 + layer.KN, "uniform")
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    ctx, sh, P = gpu_ctx, layer.shape(N), layer.P
    w = ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    if not ctx.slab_supported(w, sh):
        pytest.skip("outside the slab-fed form")
    nxt = np.resize(THRESHOLDS, N)
    img_in = api.bordered_image_bytes(N, layer.C, layer.H, layer.W, P, P)
    img_out = api.bordered_image_bytes(N, layer.KN, layer.OH, layer.OW, P, P)
    d_x, d_t, d_n = ctx.to_device(case.x), ctx.to_device(case.thr), ctx.to_device(nxt)
    d_in, d_out, d_ref = ctx.malloc(img_in), ctx.malloc(img_out), ctx.malloc(img_out)
    d_y = ctx.malloc(4 * N * layer.KN * layer.OH * layer.OW)
    try:
        ctx.quantise_e2m1_bordered(ternary, d_x, d_t, d_in, N, layer.C, layer.H, layer.W, P, P)
        ctx.gemm_slab(w, d_in, d_y, sh, alpha)
        ctx.quantise_e2m1_bordered(ternary, d_y, d_n, d_ref, N, layer.KN, layer.OH, layer.OW, P, P)
        ctx.fill(d_out, np.full(img_out, 0x77, np.uint8))
        for _ in range(2):
            ctx.gemm_slab_packed_out(w, d_in, d_out, d_n, 3 if ternary else 5, (P, P), sh, alpha)
        ctx.sync()
        want = ctx.to_host(d_ref, (img_out,), np.uint8)
        assert ctx.to_host(d_out, (img_out,), np.uint8).tobytes() == want.tobytes(), "slab-fed"
        if ternary:
            ctx.quantise_e2m1(d_x, d_t, d_in, N, layer.C, layer.H, layer.W)
            ctx.quantise_e2m1(d_y, d_n, d_ref, N, layer.KN, layer.OH, layer.OW)
            ctx.gemm_im2col_packed_out(w, d_in, d_out, d_n, 2, sh, alpha)
            ctx.sync()
            n = api.e2m1_image_bytes(N, layer.KN, layer.OH, layer.OW)
            assert ctx.to_host(d_out, (n,), np.uint8).tobytes() == ctx.to_host(d_ref, (n,), np.uint8).tobytes(), "im2col-fed"
    finally:
        for p in (d_x, d_t, d_n, d_in, d_out, d_ref, d_y):
            ctx.free(p)
        w.free()
