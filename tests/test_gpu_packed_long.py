"""GPU suite: the GEMM over an explicit packed matrix of more than 2^31 rows, past what a tensor copy's coordinates reach: its rows are
loaded by the expanders themselves.  68.8 GB of matrix, 8.6 GB of output; compared with the same rows as matrices of their own."""
import numpy as np
import pytest

import fastertnn_b200 as ft
from cases import BNN, BTN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("type_", [BNN, BTN])
def test_more_rows_than_coordinates(type_, gpu_ctx):
    import torch
    ctx = gpu_ctx
    N, OH, edge = 1 << 20, 2049, 5 * 2049  # images of 2049 x 1 pixels; the images compared at either end
    M = N * OH
    assert M > 2**31
    if ctx.mem_info()[0] < 100e9:
        pytest.skip("needs 100 GB of free device memory")
    g = np.random.default_rng(77)
    w = g.choice(np.array([-1, 1] if type_ == BNN else [-1, 0, 1], np.float32), (1, 64, 1, 1))
    pack = ft.pack_weights_binary if type_ == BNN else ft.pack_weights_ternary
    h = ctx.upload_weights(type_, pack(w, np.full(1, 0.0 if type_ == BNN else 0.5, np.float32)), 64, 1, 1)
    words = ft.k_padded(64, 1, 1)
    assert words == 4
    try:
        a = torch.zeros((M, words), dtype=torch.int64, device="cuda")  # every channel +1
        y = torch.full((M,), float("nan"), device="cuda")
        gen = torch.Generator(device="cuda").manual_seed(78)
        for rows in (a[:edge], a[M - edge:]):
            rows[:, 0] = torch.randint(-2**63, 2**63 - 1, (edge,), device="cuda", generator=gen)
        ends = [torch.empty(edge, device="cuda") for _ in range(2)]
        same = torch.empty(OH, device="cuda")
        torch.cuda.synchronize()
        ctx.gemm(h, a.data_ptr(), y.data_ptr(), N, OH, 1, 0.5)
        for rows, out in ((a[:edge], ends[0]), (a[M - edge:], ends[1])):
            ctx.gemm(h, rows.data_ptr(), out.data_ptr(), edge // OH, OH, 1, 0.5, algo=ft.GEMM_POPC_TILED)
        ctx.gemm(h, a[edge:].data_ptr(), same.data_ptr(), 1, OH, 1, 0.5, algo=ft.GEMM_POPC_TILED)
        ctx.sync()
        assert torch.equal(y[:edge], ends[0]) and torch.equal(y[M - edge:], ends[1])
        assert len(torch.unique(ends[0])) > 10 and len(torch.unique(same)) == 1
        for r in range(edge, M - edge, 1 << 28):
            assert bool((y[r:min(r + (1 << 28), M - edge)] == same[0]).all()), r
    finally:
        h.free()
        a = y = rows = out = None  # no view may keep the matrix: the tests that follow need the memory
        torch.cuda.empty_cache()
    assert ctx.mem_info()[0] > 90e9
