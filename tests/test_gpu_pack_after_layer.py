"""GPU suite: the pack kernel on a tensor that the launch in front has just written.  A layer, the pack of its output and the packed GEMM
run back to back over the same intermediate buffers with other inputs each time; every launch lets its dependents in early, so nothing
but the wait inside the pack kernel keeps it from the values of the pass before."""
import numpy as np
import pytest

import fastertnn_b200 as ft
from cases import BNN, TNN, make_case, wgt_ternary
from fastertnn_b200 import api
from fastertnn_b200.workloads import Layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("type_", [TNN, BNN])
@pytest.mark.parametrize("layout", [ft.NCHW, ft.NHWC])
@pytest.mark.parametrize("first,second,N", [(Layer(64, 12, 12, 64, 3, 3, 1, 1), Layer(64, 12, 12, 64, 3, 3, 1, 1), 2), (Layer(128, 7, 7, 512, 3, 3, 1, 1), Layer(512, 7, 7, 128, 3, 3, 1, 1), 30),
                                            (Layer(64, 9, 11, 50, 3, 3, 1, 1), Layer(50, 9, 11, 70, 3, 3, 1, 2), 6)], ids=lambda v: str(v).replace(" ", ""))
def test_pack_reads_what_the_layer_wrote(first, second, N, layout, type_, gpu_ctx, checker):
    import torch
    ctx, R, ternary = gpu_ctx, 12, type_ == TNN
    ws = []
    for L in (first, second):
        case = make_case(type_, L, 1, 9960 + L.C, "uniform")
        ws.append(ctx.upload_weights(type_, checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr), L.C, L.KH, L.KW))
    s1, s2 = first.shape(N), second.shape(N)
    gen = torch.Generator(device="cuda").manual_seed(9961)
    x = torch.empty((R, N * first.C * first.H * first.W), device="cuda").uniform_(-1, 1, generator=gen)
    t1, t2 = torch.full((N,), 0.25 if ternary else 0.0, device="cuda"), torch.full((N,), 3.25 if ternary else 0.5, device="cuda")
    mid = torch.empty(N * first.KN * first.OH * first.OW, device="cuda")
    a = torch.empty(api.packed_bytes(type_, s2), dtype=torch.uint8, device="cuda")
    y, want = (torch.full((R, N * second.KN * second.OH * second.OW), float("nan"), device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    try:
        for i in range(R):
            ctx.conv(ws[0], x[i].data_ptr(), t1.data_ptr(), mid.data_ptr(), s1, 0.5, layout)
            ctx.sync()
            ctx.conv(ws[1], mid.data_ptr(), t2.data_ptr(), want[i].data_ptr(), s2, 0.5, layout, pack_algo=api.PACK_GATHER, gemm_algo=api.GEMM_POPC_TILED)
            ctx.sync()
        assert len(np.unique(want[0].cpu().numpy())) > 10
        for rep in range(4):
            for i in range(R):
                ctx.conv(ws[0], x[i].data_ptr(), t1.data_ptr(), mid.data_ptr(), s1, 0.5, layout)
                ctx.pack(ternary, mid.data_ptr(), t2.data_ptr(), a.data_ptr(), s2, layout)
                ctx.gemm(ws[1], a.data_ptr(), y[i].data_ptr(), N, second.OH, second.OW, 0.5, layout)
            ctx.sync()
            assert torch.equal(y, want), rep
            y.fill_(float("nan"))
            torch.cuda.synchronize()
    finally:
        for w in ws:
            w.free()
