"""GPU suite: image outputs whose slabs the loaders fetch, over the depths of the slab ring -- eight, six, four and two slabs beside
resident weights (two MMA issuers), large slabs and several tiles per block, with slopes inside and outside (0, 1]."""
import numpy as np
import pytest

from cases import BNN, BTN, TBN, TNN, make_case, wgt_ternary
from fastertnn_b200 import api
from fastertnn_b200.workloads import Layer

pytestmark = pytest.mark.gpu

LAYERS = [
    (Layer(128, 64, 64, 64, 3, 3, 1, 1), 14), (Layer(128, 132, 132, 64, 3, 3, 1, 1), 4), (Layer(128, 16, 200, 64, 3, 3, 1, 1), 20),
    (Layer(128, 12, 340, 50, 3, 3, 1, 1), 14), (Layer(64, 12, 256, 64, 3, 3, 1, 1), 19), (Layer(128, 64, 64, 128, 3, 3, 1, 1), 14),
    (Layer(128, 12, 300, 100, 3, 3, 1, 1), 14), (Layer(64, 40, 80, 128, 5, 5, 2, 1), 18), (Layer(128, 12, 12, 256, 3, 3, 1, 1), 70),
]


@pytest.mark.parametrize("type_,alpha", [(TNN, 0.5), (TBN, 1.5), (BTN, -0.25), (BNN, 0.3)])
@pytest.mark.parametrize("layer,N", LAYERS, ids=lambda v: str(v).replace(" ", ""))
def test_loader_ring_depths(layer, N, type_, alpha, gpu_ctx, checker):
    ternary = type_ in (TNN, TBN)
    case = make_case(type_, layer, N, 9970 + layer.KN, "uniform")
    ctx, sh, P = gpu_ctx, layer.shape(N), layer.P
    w = ctx.upload_weights(type_, checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr), layer.C, layer.KH, layer.KW)
    assert ctx.slab_supported(w, sh)
    nxt = np.resize(np.array([0.25, -1.0, 3.5], np.float32), N)
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
        assert ctx.to_host(d_out, (img_out,), np.uint8).tobytes() == ctx.to_host(d_ref, (img_out,), np.uint8).tobytes()
    finally:
        for p in (d_x, d_t, d_n, d_in, d_out, d_ref, d_y):
            ctx.free(p)
        w.free()
