"""GPU suite: a wait that runs out inside a whole layer kernel ends the launch with the status word set.  The one-launch slab form is
started with quantiser warps that are told of no image: its producers wait for images that never come, give up after about a second,
and every role of every block has to leave (the producer is one lane of its warp, so its warp barriers must pair up on that path too)."""
import numpy as np
import pytest

import fastertnn_b200 as ft
from cases import TNN, make_case, wgt_ternary
from fastertnn_b200 import api
from fastertnn_b200.workloads import Layer

pytestmark = pytest.mark.gpu


# 32-byte pixels with weights that stay, 128-byte pixels with streamed ones, block pairs
@pytest.mark.parametrize("layer,N,pairs", [(Layer(64, 12, 12, 64, 3, 3, 1, 1), 5, 1), (Layer(256, 10, 10, 128, 3, 3, 1, 1), 3, 1),
                                           (Layer(256, 14, 14, 256, 3, 3, 1, 1), 4, 2)], ids=lambda v: str(v).replace(" ", ""))
def test_expired_producer_wait_leaves_the_layer_kernel(layer, N, pairs, gpu_ctx, checker):
    ctx, sh = gpu_ctx, layer.shape(N)
    case = make_case(TNN, layer, N, 9950 + layer.C, "uniform")
    wp = checker.pack_weights(wgt_ternary(TNN), case.w, case.w_thr)
    want = checker.conv(TNN, case.x, case.thr, wp, case.kernel_hw, case.padding, case.stride, case.alpha)
    w = ctx.upload_weights(TNN, wp, layer.C, layer.KH, layer.KW)
    nb = api.slab_workspace_bytes(N, layer.C, layer.H, layer.W, layer.P, layer.P)
    d_x, d_t, d_ws, d_y = ctx.to_device(case.x), ctx.to_device(case.thr), ctx.malloc(nb), ctx.malloc(want.nbytes)
    try:
        stale = np.full(want.shape, 7.5, np.float32)
        ctx.fill(d_y, stale)
        api._check(ctx.lib.tnns_cuda_selftest_slab_wait_expiry(ctx.handle, w.handle, d_x, d_t, d_y, d_ws, nb, sh, pairs, 0))
        with pytest.raises(ft.TnnsError) as e:
            ctx.sync()
        assert e.value.status == 5 and "wait" in e.value.detail
        assert ctx.to_host(d_y, want.shape, np.float32).tobytes() == stale.tobytes()
        for _ in range(2):  # the synchronisation words were left clean
            ctx.conv_slab(w, d_x, d_t, d_y, d_ws, nb, sh, case.alpha, pairs)
        ctx.sync()
        assert ctx.to_host(d_y, want.shape, np.float32).tobytes() == want.tobytes()
    finally:
        for p in (d_x, d_t, d_ws, d_y):
            ctx.free(p)
        w.free()
