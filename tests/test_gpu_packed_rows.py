"""GPU suite: the 4-bit GEMM over an explicit packed matrix, whose rows arrive as tensor copies, against the integer-pipe kernel."""
import numpy as np
import pytest

import fastertnn_b200 as ft
from cases import BNN, BTN, TBN, TNN, make_case, wgt_ternary
from fastertnn_b200 import api
from fastertnn_b200.workloads import Layer

pytestmark = pytest.mark.gpu

# one row, row counts around the tile, fewer stages than groups, odd numbers of stages, more stages than any ring, kernel counts around
# the tiles, several tiles per block
LAYERS = [
    (Layer(64, 1, 1, 64, 1, 1, 0, 1), 1), (Layer(300, 1, 1, 65, 1, 1, 0, 1), 127), (Layer(700, 1, 1, 257, 1, 1, 0, 1), 129),
    (Layer(64, 9, 9, 20, 3, 3, 1, 1), 4), (Layer(192, 8, 8, 128, 3, 3, 1, 1), 5), (Layer(130, 12, 12, 129, 5, 3, 1, 2), 8),
    (Layer(64, 40, 40, 64, 3, 3, 1, 1), 30), (Layer(256, 24, 24, 300, 1, 1, 0, 1), 70), (Layer(512, 6, 6, 512, 3, 3, 1, 1), 9),
]


@pytest.mark.parametrize("type_", [TNN, TBN, BTN, BNN])
@pytest.mark.parametrize("layer,N", LAYERS, ids=lambda v: str(v).replace(" ", ""))
def test_packed_rows(layer, N, type_, gpu_ctx, checker):
    ternary = type_ in (TNN, TBN)
    case = make_case(type_, layer, N, 9600 + layer.KN, "uniform")
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    ctx, sh = gpu_ctx, layer.shape(N)
    w = ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    n_out = N * layer.KN * layer.OH * layer.OW
    d_x, d_t = ctx.to_device(case.x), ctx.to_device(case.thr)
    d_a, d_y, d_r = ctx.malloc(api.packed_bytes(type_, sh)), ctx.malloc(4 * n_out), ctx.malloc(4 * n_out)
    try:
        ctx.pack(ternary, d_x, d_t, d_a, sh)
        for layout in (ft.NCHW, ft.NHWC):
            ctx.fill(d_y, np.full(n_out, np.nan, np.float32))
            ctx.gemm(w, d_a, d_r, N, layer.OH, layer.OW, case.alpha, layout, algo=api.GEMM_POPC_TILED)
            for _ in range(2):
                ctx.gemm(w, d_a, d_y, N, layer.OH, layer.OW, case.alpha, layout, algo=api.GEMM_F4_TC)
            ctx.sync()
            assert ctx.to_host(d_y, (n_out,), np.float32).tobytes() == ctx.to_host(d_r, (n_out,), np.float32).tobytes(), layout
    finally:
        for p in (d_x, d_t, d_a, d_y, d_r):
            ctx.free(p)
        w.free()


# many stages on tiles of 256 kernels: a slot of the packed-row ring is read while its refill is on the way, so every launch has to be
# right, beside others and alone (a row read too late holds the next lap's bytes in a few launches of a hundred)
@pytest.mark.parametrize("type_,layer,N", [(TNN, Layer(512, 14, 14, 512, 3, 3, 1, 1), 64), (TNN, Layer(512, 7, 7, 512, 3, 3, 1, 1), 256),
                                           (BTN, Layer(1024, 7, 7, 512, 3, 3, 1, 1), 100), (BNN, Layer(512, 7, 7, 64, 3, 3, 1, 1), 100)],
                         ids=lambda v: str(v).replace(" ", ""))
def test_every_launch_of_many(type_, layer, N, gpu_ctx, checker):
    import torch
    ctx, sh, R = gpu_ctx, layer.shape(N), 6
    case = make_case(type_, layer, 1, 9700 + layer.C, "uniform")
    w = ctx.upload_weights(type_, checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr), layer.C, layer.KH, layer.KW)
    ternary = type_ in (TNN, TBN)
    gen = torch.Generator(device="cuda").manual_seed(9701)
    n_out = N * layer.KN * layer.OH * layer.OW
    x = torch.empty(N * layer.C * layer.H * layer.W, device="cuda")
    t = torch.full((N,), 0.25 if ternary else 0.0, device="cuda")
    a = torch.empty((R, api.packed_bytes(type_, sh) // 8), dtype=torch.int64, device="cuda")
    y, want = torch.empty((R, n_out), device="cuda"), torch.empty((R, n_out), device="cuda")
    try:
        for i in range(R):
            x.uniform_(-1, 1, generator=gen)
            torch.cuda.synchronize()
            ctx.pack(ternary, x.data_ptr(), t.data_ptr(), a[i].data_ptr(), sh)
            ctx.gemm(w, a[i].data_ptr(), want[i].data_ptr(), N, layer.OH, layer.OW, case.alpha, algo=api.GEMM_POPC_TILED)
            ctx.sync()
        wrong = 0
        for rep in range(60):
            y.fill_(float("nan"))
            torch.cuda.synchronize()
            for i in range(R):
                ctx.gemm(w, a[i].data_ptr(), y[i].data_ptr(), N, layer.OH, layer.OW, case.alpha, algo=api.GEMM_F4_TC)
                if rep % 2:
                    ctx.sync()
            ctx.sync()
            wrong += int((y != want).any(1).sum())
        assert wrong == 0, f"{wrong} of {60 * R} launches"
    finally:
        w.free()
