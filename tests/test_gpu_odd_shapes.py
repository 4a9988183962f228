"""GPU suite: layers of sizes that are no multiple of anything.  The quantise kernels that read with plain
loads (unaligned rows, unaligned bases, tiny tensors) against a numpy construction of their images, and whole
layers with ragged channel counts or binary activations and strides against the checker."""
import numpy as np
import pytest

import fastertnn_b200 as ft
from cases import BNN, BTN, TBN, TNN, make_case, to_nchw, to_nhwc, wgt_ternary
from fastertnn_b200 import synth
from fastertnn_b200.workloads import Layer
from test_gpu_parity import _expand32_f4_numpy

pytestmark = pytest.mark.gpu


def numpy_planes(x, thr, tern):
    """[n][plane][pixel][ic][lo, hi] uint32 of an fp32 NCHW tensor, by the reference's compares."""
    N, C, H, W = x.shape
    Cp = (C + 63) // 64
    t = thr.reshape(N, 1, 1)
    v = x.reshape(N, C, H * W)
    bits = np.zeros((2 if tern else 1, N, Cp * 64, H * W), bool)
    bits[0, :, :C] = v < (-t if tern else t)
    if tern:
        bits[1] = True
        bits[1, :, :C] = ~((v < -t) | (v > t))
    packed = np.ascontiguousarray(np.packbits(bits.transpose(1, 0, 3, 2), axis=-1, bitorder="little"))   # n, plane, pixel, channel bits
    return packed.view(np.uint32).reshape(N, 2 if tern else 1, H * W, Cp, 2)


@pytest.mark.parametrize("tern", [True, False])
@pytest.mark.parametrize("N,C,H,W", [(1, 1, 1, 1), (3, 33, 1, 1), (1, 64, 5, 5), (5, 65, 7, 3), (2, 31, 31, 33), (33, 130, 1, 7), (4, 262, 9, 5), (7, 3, 15, 23),
                                     (2, 64, 8, 8), (3, 192, 6, 6), (2, 8, 7, 5), (2, 9, 7, 5), (2, 16, 7, 5), (2, 17, 7, 5), (2, 24, 7, 5), (2, 25, 7, 5), (2, 126, 7, 5)])
def test_quantise_with_plain_loads(N, C, H, W, tern, gpu_ctx):
    """One pixel, one channel, tails on both sides of 32 and 64 channels, pixel counts around 32, warps that straddle
    images; and sizes the copy engine would take, from a base that is not 16-byte aligned."""
    ctx = gpu_ctx
    x = synth.uniform_pm1(300 + C, (N, C, H, W))
    thr = (synth.uniform_pm1(301, (N,)) * 0.3 + (0.2 if tern else 0.0)).astype(np.float32)
    flat = x.reshape(-1)
    flat[:: 5] = np.float32(0.0)
    flat[1:: 7] = np.repeat(thr, C * H * W)[1:: 7]       # exactly on the threshold: compares are strict
    want = numpy_planes(x, thr, tern)
    want4 = _expand32_f4_numpy(want[:, 0], want[:, 1]) if tern else None
    Cp = (C + 63) // 64
    nb_p, nb_e = ft.api.packed_image_bytes(tern, N, C, H, W), ft.api.e2m1_image_bytes(N, C, H, W)
    d_t, d_p, d_e, d_x = ctx.to_device(thr), ctx.malloc(nb_p), ctx.malloc(nb_e), ctx.malloc(x.nbytes + 16)
    try:
        for layout in (ft.NCHW, ft.NHWC):
            for off in (0, 4):
                ctx.fill(d_x + off, x if layout == ft.NCHW else to_nhwc(x))
                ctx.fill(d_p, np.full(nb_p // 4, 0x5A5A5A5A, np.uint32))
                ctx.quantise(tern, d_x + off, d_t, d_p, N, C, H, W, layout)
                ctx.sync()
                assert np.array_equal(ctx.to_host(d_p, want.shape, np.uint32), want), ("planes", layout, off)
                if tern:
                    ctx.fill(d_e, np.full(nb_e // 4, 0x5A5A5A5A, np.uint32))
                    ctx.quantise_e2m1(d_x + off, d_t, d_e, N, C, H, W, layout)
                    ctx.sync()
                    assert np.array_equal(ctx.to_host(d_e, (N, H * W, Cp, 2, 4), np.uint32), want4), ("4-bit image", layout, off)
    finally:
        for p in (d_t, d_p, d_e, d_x):
            ctx.free(p)


# ragged channel counts (pixels of 96, 160, 192, 224 bytes of operands), binary activations with strides and paddings,
# pad-to-four words under binary weights, odd images: layers whose image is stored padded or bordered for the copy engine
WIDE_LAYERS = [
    (Layer(130, 9, 7, 40, 3, 3, 1, 1), 3), (Layer(320, 15, 23, 300, 3, 3, 1, 2), 2), (Layer(384, 5, 5, 64, 1, 1, 0, 1), 3),
    (Layer(420, 6, 6, 129, 5, 3, 2, 2), 2), (Layer(600, 1, 1, 70, 1, 1, 0, 1), 5), (Layer(64, 12, 12, 64, 3, 3, 1, 2), 3),
    (Layer(128, 9, 9, 33, 3, 3, 1, 3), 3), (Layer(256, 14, 14, 256, 3, 3, 1, 2), 3), (Layer(40, 7, 7, 20, 3, 3, 0, 1), 4),
    (Layer(96, 8, 8, 200, 2, 2, 3, 1), 2), (Layer(70, 5, 5, 16, 1, 1, 0, 2), 7), (Layer(512, 4, 4, 40, 3, 3, 1, 1), 5),
]


@pytest.mark.parametrize("type_", [TNN, TBN, BTN, BNN])
@pytest.mark.parametrize("layer,N", WIDE_LAYERS, ids=lambda v: str(v).replace(" ", ""))
def test_layers_of_any_channel_count_and_alphabet(layer, N, type_, gpu_ctx, checker):
    """Whole layers through the default call, both layouts, twice over stale workspaces."""
    case = make_case(type_, layer, N, 8200 + layer.C, "uniform")
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    want = checker.conv(type_, case.x, case.thr, wp, case.kernel_hw, case.padding, case.stride, case.alpha)
    ctx = gpu_ctx
    w = ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    d_t, d_y = ctx.to_device(case.thr), ctx.malloc(want.nbytes)
    nb = -(-ctx.conv_workspace_bytes(w, layer.shape(N)) // 4) * 4
    d_ws = ctx.malloc(nb)
    try:
        for layout in (ft.NCHW, ft.NHWC):
            d_x = ctx.to_device(case.x if layout == ft.NCHW else to_nhwc(case.x))
            for fill in (0x77777777, 0xFFFFFFFF):
                ctx.fill(d_ws, np.full(nb // 4, fill, np.uint32))
                ctx.fill(d_y, np.full(want.size, np.nan, np.float32))
                ctx.conv_ws(w, d_x, d_t, d_y, d_ws, nb, layer.shape(N), case.alpha, layout)
                ctx.sync()
                got = ctx.to_host(d_y, want.shape if layout == ft.NCHW else (N, layer.OH, layer.OW, layer.KN), np.float32)
                got = got if layout == ft.NCHW else to_nchw(got)
                assert got.tobytes() == want.tobytes(), (layout, fill)
            ctx.free(d_x)
    finally:
        for p in (d_t, d_y, d_ws):
            ctx.free(p)
        w.free()


@pytest.mark.parametrize("layer,N", [(Layer(130, 20, 20, 400, 3, 3, 1, 1), 75), (Layer(192, 24, 24, 368, 3, 3, 1, 1), 52)], ids=lambda v: str(v).replace(" ", ""))
def test_ragged_channels_in_one_launch(layer, N, gpu_ctx, checker):
    """Enough tiles for the form that quantises inside the GEMM launch, with pixels padded to whole stage rows."""
    from cases import threaded_conv
    case = make_case(TNN, layer, N, 8300, "uniform")
    wp = checker.pack_weights(True, case.w, case.w_thr)
    want = threaded_conv(checker, TNN, case.x, case.thr, wp, layer)
    ctx = gpu_ctx
    w = ctx.upload_weights(TNN, wp, layer.C, layer.KH, layer.KW)
    d_t, d_x, d_y = ctx.to_device(case.thr), ctx.to_device(case.x), ctx.malloc(want.nbytes)
    try:
        before = ft.api.launch_count()
        ctx.conv(w, d_x, d_t, d_y, layer.shape(N), case.alpha)
        assert ft.api.launch_count() - before == 1
        ctx.sync()
        assert ctx.to_host(d_y, want.shape, np.float32).tobytes() == want.tobytes()
    finally:
        for p in (d_t, d_x, d_y):
            ctx.free(p)
        w.free()


# tiles of 128 rows x 256 kernels on either side of three per SM (148 SMs); the form that quantises inside the GEMM launch fetches
# pixel-major rows in 16-byte multiples, so C % 4 decides between one launch and two
@pytest.mark.parametrize("type_,layer,N,launches", [
    (TNN, Layer(262, 21, 20, 512, 3, 3, 1, 1), 70, 2), (TNN, Layer(262, 21, 20, 512, 3, 3, 1, 1), 63, 2), (TBN, Layer(130, 20, 20, 400, 3, 3, 1, 1), 75, 2),
    (TNN, Layer(390, 14, 14, 512, 3, 3, 1, 1), 150, 2), (TNN, Layer(262, 1, 1, 4096, 1, 1, 0, 1), 4000, 2), (TNN, Layer(132, 20, 20, 400, 3, 3, 1, 1), 75, 1),
    (TBN, Layer(192, 24, 24, 368, 3, 3, 1, 1), 52, 1), (TNN, Layer(192, 24, 24, 368, 3, 3, 1, 1), 48, 2)], ids=lambda v: str(v).replace(" ", ""))
def test_ragged_channels_pixel_major(type_, layer, N, launches, gpu_ctx, checker):
    from cases import threaded_conv
    case = make_case(type_, layer, N, 8400 + layer.C, "uniform")
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    want = threaded_conv(checker, type_, case.x, case.thr, wp, layer)
    ctx = gpu_ctx
    w = ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    d_t, d_x, d_y = ctx.to_device(case.thr), ctx.to_device(to_nhwc(case.x)), ctx.malloc(want.nbytes)
    try:
        for _ in range(2):
            ctx.fill(d_y, np.full(want.size, np.nan, np.float32))
            before = ft.api.launch_count()
            ctx.conv(w, d_x, d_t, d_y, layer.shape(N), case.alpha, ft.NHWC)
            assert ft.api.launch_count() - before == launches
            ctx.sync()
            assert to_nchw(ctx.to_host(d_y, (N, layer.OH, layer.OW, layer.KN), np.float32)).tobytes() == want.tobytes()
    finally:
        for p in (d_t, d_x, d_y):
            ctx.free(p)
        w.free()


@pytest.mark.parametrize("type_", [BTN, BNN])
def test_im2col_calls_refuse_binary_activations(type_, gpu_ctx, checker):
    """Unpadded layers too, whose geometry alone would fit: the 4-bit image these calls read is a ternary one."""
    layer, N = Layer(200, 8, 8, 160, 1, 1, 0, 1), 3
    case = make_case(type_, layer, N, 8500, "uniform")
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    ctx, shape = gpu_ctx, layer.shape(N)
    w = ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    d_t, d_img = ctx.to_device(case.thr), ctx.malloc(ft.api.e2m1_image_bytes(N, layer.C, layer.H, layer.W))
    d_y = ctx.malloc(4 * N * layer.KN * layer.OH * layer.OW)
    try:
        assert not ctx.im2col_supported(w, shape)
        calls = [lambda: ctx.gemm_im2col(w, d_img, d_y, shape, 0.5), lambda: ctx.gemm_im2col_bordered_out(w, d_img, d_y, d_t, (1, 1), shape, 0.5)]
        calls += [lambda f=f: ctx.gemm_im2col_packed_out(w, d_img, d_y, d_t, f, shape, 0.5) for f in (0, 1, 2)]
        for call in calls:
            with pytest.raises(ft.TnnsError) as e:
                call()
            assert e.value.status == 4
    finally:
        for p in (d_t, d_img, d_y):
            ctx.free(p)
        w.free()


def test_ragged_channels_first_call_inside_a_capture(gpu_ctx, checker):
    """A context whose first call of the layer is recorded into a graph: nothing may be allocated there, and the graph keeps no
    state of the context's (it is replayed on another stream than it was recorded on)."""
    import torch
    from cases import threaded_conv
    layer, N = Layer(130, 20, 20, 400, 3, 3, 1, 1), 75
    case = make_case(TNN, layer, N, 8700, "uniform")
    wp = checker.pack_weights(True, case.w, case.w_thr)
    want = threaded_conv(checker, TNN, case.x, case.thr, wp, layer)
    ctx, nb = ft.Context(0), 32 << 20
    w = ctx.upload_weights(TNN, wp, layer.C, layer.KH, layer.KW)
    d_t, d_x, d_y, d_ws = ctx.to_device(case.thr), ctx.to_device(case.x), ctx.malloc(want.nbytes), ctx.malloc(nb)
    try:
        s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            ctx.conv_ws(w, d_x, d_t, d_y, d_ws, nb, layer.shape(N), case.alpha, ft.NCHW, ft.PACK_AUTO, ft.GEMM_AUTO, s.cuda_stream)
        for rep in range(2):
            ctx.fill(d_y, np.full(want.size, np.nan, np.float32))
            graph.replay()
            torch.cuda.synchronize()
            assert ctx.to_host(d_y, want.shape, np.float32).tobytes() == want.tobytes(), rep
    finally:
        for p in (d_t, d_x, d_y, d_ws):
            ctx.free(p)
        w.free()
        ctx.close()


@pytest.mark.parametrize("type_,layer,N,layout,offset", [
    (TNN, Layer(64, 31, 33, 64, 3, 3, 1, 1), 2, ft.NCHW, 0), (TNN, Layer(64, 32, 32, 64, 3, 3, 1, 1), 2, ft.NCHW, 4), (TBN, Layer(70, 20, 20, 96, 3, 3, 1, 1), 2, ft.NHWC, 0),
    (BTN, Layer(256, 15, 17, 64, 3, 3, 1, 1), 2, ft.NCHW, 0), (BNN, Layer(128, 1, 1, 64, 1, 1, 0, 1), 5, ft.NHWC, 4)], ids=lambda v: str(v).replace(" ", ""))
def test_the_reported_algorithm_can_be_asked_for(type_, layer, N, layout, offset, gpu_ctx, checker):
    """Inputs the copy engine cannot fetch: what conv_auto_algo answers is what the call takes, by itself and on request."""
    case = make_case(type_, layer, N, 8600 + layer.C, "uniform")
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    want = checker.conv(type_, case.x, case.thr, wp, case.kernel_hw, case.padding, case.stride, case.alpha)
    ctx, shape = gpu_ctx, layer.shape(N)
    w = ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    d_t, d_y, base = ctx.to_device(case.thr), ctx.malloc(want.nbytes), ctx.malloc(case.x.nbytes + 16)
    d_x = base + offset
    try:
        ctx.fill(d_x, case.x if layout == ft.NCHW else to_nhwc(case.x))
        algo = ctx.conv_auto_algo(w, shape, d_x, layout)
        assert algo == ft.GEMM_F4_SLAB
        for how in (ft.GEMM_AUTO, algo):
            ctx.fill(d_y, np.full(want.size, np.nan, np.float32))
            ctx.conv(w, d_x, d_t, d_y, shape, case.alpha, layout, ft.PACK_AUTO, how)
            ctx.sync()
            got = ctx.to_host(d_y, want.shape if layout == ft.NCHW else (N, layer.OH, layer.OW, layer.KN), np.float32)
            assert (got if layout == ft.NCHW else to_nchw(got)).tobytes() == want.tobytes(), how
        # the one launch reads through the copy engine: still refused
        with pytest.raises(ft.TnnsError) as e:
            ctx.conv(w, d_x, d_t, d_y, shape, case.alpha, layout, ft.PACK_AUTO, ft.GEMM_F4_SLAB_FUSED)
        assert e.value.status == 4
    finally:
        for p in (d_t, d_y, base):
            ctx.free(p)
        w.free()


@pytest.mark.parametrize("type_", [TNN, TBN, BTN, BNN])
@pytest.mark.parametrize("layer,N", WIDE_LAYERS + [(Layer(320, 12, 12, 64, 1, 1, 0, 1), 2), (Layer(3, 12, 12, 64, 3, 3, 1, 1), 2), (Layer(64, 30, 30, 64, 3, 3, 1, 1), 1)],
                         ids=lambda v: str(v).replace(" ", ""))
def test_workspace_of_the_queried_size_holds_every_route(layer, N, type_, gpu_ctx, checker):
    """conv_ws in exactly conv_workspace_bytes() bytes writes the image of the route conv() takes, not that of one with a smaller
    workspace, and nothing past them."""
    case = make_case(type_, layer, N, 8900 + layer.C, "uniform")
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    want = checker.conv(type_, case.x, case.thr, wp, case.kernel_hw, case.padding, case.stride, case.alpha)
    ctx, shape = gpu_ctx, layer.shape(N)
    w = ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    nb = ctx.conv_workspace_bytes(w, shape)
    tern, cp = type_ in (TNN, TBN), (layer.C + 63) // 64
    assert nb >= ft.api.packed_image_bytes(tern, N, layer.C, layer.H, layer.W)
    if ctx.im2col_supported(w, shape):
        assert nb >= ft.api.fused_workspace_bytes(N, layer.C, layer.H, layer.W)
    if ctx.slab_supported(w, shape):
        assert nb >= ft.api.slab_workspace_bytes(N, layer.C, layer.H, layer.W, layer.P, layer.P)
    if ctx.dense_supported(w, shape):
        assert nb >= ft.api.dense_workspace_bytes(shape)
    assert ctx.conv_workspace_bytes(w, Layer(layer.C + 1, layer.H, layer.W, layer.KN, layer.KH, layer.KW, layer.P, layer.S).shape(N)) == 0
    guard = 4096
    d_t, d_x, d_y, d_ws = ctx.to_device(case.thr), ctx.to_device(case.x), ctx.malloc(want.nbytes), ctx.malloc((nb + 3) // 4 * 4 + guard)
    try:
        ctx.fill(d_ws, np.full((nb + 3) // 4 + guard // 4, 0x55555555, np.uint32))   # no 4-bit operand is a 5
        ctx.fill(d_y, np.full(want.size, np.nan, np.float32))
        ctx.conv_ws(w, d_x, d_t, d_y, d_ws, nb, shape, case.alpha)
        ctx.sync()
        assert ctx.to_host(d_y, want.shape, np.float32).tobytes() == want.tobytes()
        ws = ctx.to_host(d_ws, ((nb + 3) // 4 * 4 + guard,), np.uint8)
        assert (ws[nb:] == 0x55).all(), "past the workspace"
        if ctx.conv_auto_algo(w, shape, d_x) != ft.GEMM_F4_DENSE:
            border = layer.P if not tern or ctx.conv_auto_algo(w, shape, d_x) == ft.GEMM_F4_SLAB else 0
            pitch = 32 * (cp if cp <= 2 else -(-cp // 4) * 4)
            last = N * (layer.H + 2 * border) * (layer.W + 2 * border) * pitch - pitch   # the last pixel of the 4-bit image
            px = ws[last:last + 32 * cp]
            assert np.isin(px & 15, (0, 2, 10)).all() and np.isin(px >> 4, (0, 2, 10)).all()
    finally:
        for p in (d_t, d_x, d_y, d_ws):
            ctx.free(p)
        w.free()


@pytest.mark.parametrize("type_", [TNN, TBN])
def test_ragged_channels_in_one_launch_on_two_streams(type_, checker):
    """The context's own synchronisation words serve the stream that came first, the words behind the image any other one."""
    import torch
    from cases import threaded_conv
    layer, N = Layer(130, 20, 20, 400, 3, 3, 1, 1), 75
    case = make_case(type_, layer, N, 8350, "uniform")
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    want = threaded_conv(checker, type_, case.x, case.thr, wp, layer)
    ctx = ft.Context(0)
    w = ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    shape = layer.shape(N)
    nb = ctx.conv_workspace_bytes(w, shape)
    d_t, d_x = ctx.to_device(case.thr), ctx.to_device(case.x)
    d_y, d_ws = [ctx.malloc(want.nbytes) for _ in range(2)], [ctx.malloc(nb) for _ in range(2)]
    side = torch.cuda.Stream()
    streams = [0, side.cuda_stream]
    try:
        for k in range(2):
            ctx.fill(d_y[k], np.full(want.size, np.nan, np.float32))
            ctx.fill(d_ws[k], np.full(nb // 4, 0xFFFFFFFF, np.uint32))
        before = ft.api.launch_count()
        for rep in range(3):
            for k in range(2):
                ctx.conv_ws(w, d_x, d_t, d_y[k], d_ws[k], nb, shape, case.alpha, ft.NCHW, ft.PACK_AUTO, ft.GEMM_AUTO, streams[k])
        assert ft.api.launch_count() - before == 6, "one launch each"
        torch.cuda.synchronize()
        ctx.sync()
        for k in range(2):
            assert ctx.to_host(d_y[k], want.shape, np.float32).tobytes() == want.tobytes(), k
        # a workspace too small for the words behind the image: two launches
        ctx.conv_ws(w, d_x, d_t, d_y[0], d_ws[0], nb - 128, shape, case.alpha)
        ctx.sync()
        assert ctx.to_host(d_y[0], want.shape, np.float32).tobytes() == want.tobytes()
        assert ft.api.launch_count() - before == 8
    finally:
        for p in [d_t, d_x] + d_y + d_ws:
            ctx.free(p)
        w.free()
        ctx.close()


def with_special_values(x, thr, nan=False):
    """Every third value one where a quantiser can go wrong: +-0, +-threshold and the floats beside it, denormals, infinities."""
    f = np.float32
    specials = []
    for t in np.unique(np.abs(thr)):
        for s in (f(t), f(-t)):
            specials += [s, np.nextafter(s, f(np.inf)), np.nextafter(s, f(-np.inf))]
    specials += [f(0.0), f(-0.0), f(1e-45), f(-1e-45), f(1e-39), f(-1e-39), f(np.inf), f(-np.inf), f(3e38), f(-3e38)] + ([f(np.nan), -f(np.nan)] if nan else [])
    flat = x.reshape(-1)
    flat[::3] = np.resize(np.array(specials, f), flat[::3].size)
    return x


SPECIAL_THR = np.array([0.25, 0.0, -0.0, 0.75], np.float32)


@pytest.mark.parametrize("tern", [True, False])
@pytest.mark.parametrize("C,H,W", [(40, 7, 7), (96, 8, 8), (65, 5, 9), (192, 6, 6)])
def test_quantise_special_values(C, H, W, tern, gpu_ctx):
    """Plain-load and copy-engine fed kernels, full and ragged channel groups, both layouts; NaN is a ternary zero, a binary +1."""
    ctx, N = gpu_ctx, 4
    x = with_special_values(synth.uniform_pm1(400 + C, (N, C, H, W)), SPECIAL_THR, nan=True)
    want = numpy_planes(x, SPECIAL_THR, tern)
    nb_p, nb_e = ft.api.packed_image_bytes(tern, N, C, H, W), ft.api.e2m1_image_bytes(N, C, H, W)
    d_t, d_p, d_e = ctx.to_device(SPECIAL_THR), ctx.malloc(nb_p), ctx.malloc(nb_e)
    try:
        for layout in (ft.NCHW, ft.NHWC):
            d_x = ctx.to_device(x if layout == ft.NCHW else to_nhwc(x))
            ctx.quantise(tern, d_x, d_t, d_p, N, C, H, W, layout)
            ctx.sync()
            assert np.array_equal(ctx.to_host(d_p, want.shape, np.uint32), want), layout
            if tern:
                ctx.quantise_e2m1(d_x, d_t, d_e, N, C, H, W, layout)
                ctx.sync()
                want4 = _expand32_f4_numpy(want[:, 0], want[:, 1])
                assert np.array_equal(ctx.to_host(d_e, want4.shape, np.uint32), want4), ("4-bit image", layout)
            ctx.free(d_x)
    finally:
        for p in (d_t, d_p, d_e):
            ctx.free(p)


# the dense form, pixels stored padded, images stored bordered, and the plain image from plain loads
@pytest.mark.parametrize("type_,layer", [
    (TNN, Layer(3, 18, 21, 40, 7, 7, 3, 2)), (TBN, Layer(4, 9, 9, 33, 3, 3, 1, 1)), (TNN, Layer(130, 7, 7, 40, 3, 3, 1, 1)), (TBN, Layer(192, 8, 8, 64, 3, 3, 1, 2)),
    (BTN, Layer(130, 7, 7, 40, 3, 3, 1, 2)), (BNN, Layer(96, 9, 9, 70, 3, 3, 1, 2)), (TNN, Layer(256, 7, 7, 64, 3, 3, 1, 2))], ids=lambda v: str(v).replace(" ", ""))
def test_layers_with_special_values(type_, layer, gpu_ctx, checker):
    case = make_case(type_, layer, 4, 8800 + layer.C, "uniform")
    case.thr[:] = SPECIAL_THR
    with_special_values(case.x, SPECIAL_THR)
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    want = checker.conv(type_, case.x, case.thr, wp, case.kernel_hw, case.padding, case.stride, case.alpha)
    ctx = gpu_ctx
    w = ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    d_t, d_y = ctx.to_device(case.thr), ctx.malloc(want.nbytes)
    try:
        for layout in (ft.NCHW, ft.NHWC):
            d_x = ctx.to_device(case.x if layout == ft.NCHW else to_nhwc(case.x))
            ctx.conv(w, d_x, d_t, d_y, layer.shape(4), case.alpha, layout)
            ctx.sync()
            got = ctx.to_host(d_y, want.shape if layout == ft.NCHW else (4, layer.OH, layer.OW, layer.KN), np.float32)
            assert (got if layout == ft.NCHW else to_nchw(got)).tobytes() == want.tobytes(), layout
            ctx.free(d_x)
    finally:
        for p in (d_t, d_y):
            ctx.free(p)
        w.free()



# narrow and wide tiles of every GEMM: odd and even kernel counts (ragged last pairs), row bases that hold no pair or quad of floats
@pytest.mark.parametrize("type_,layer,N", [
    (TNN, Layer(64, 20, 20, 25, 3, 3, 1, 1), 30), (TNN, Layer(256, 14, 14, 101, 3, 3, 1, 1), 60), (BNN, Layer(128, 20, 20, 1, 3, 3, 1, 1), 5), (BTN, Layer(64, 20, 20, 64, 3, 3, 1, 1), 9),
    (TBN, Layer(64, 15, 15, 127, 3, 3, 1, 2), 7), (TNN, Layer(3, 30, 30, 33, 3, 3, 1, 1), 40), (TNN, Layer(256, 14, 14, 300, 1, 1, 0, 1), 60)], ids=lambda v: str(v).replace(" ", ""))
def test_pixel_major_rows_of_any_width_and_alignment(type_, layer, N, gpu_ctx, checker):
    case = make_case(type_, layer, N, 9000 + layer.C, "uniform")
    wp = checker.pack_weights(wgt_ternary(type_), case.w, case.w_thr)
    want = to_nhwc(checker.conv(type_, case.x, case.thr, wp, case.kernel_hw, case.padding, case.stride, case.alpha))
    ctx = gpu_ctx
    w = ctx.upload_weights(type_, wp, layer.C, layer.KH, layer.KW)
    d_t, d_x, d_y = ctx.to_device(case.thr), ctx.to_device(to_nhwc(case.x)), ctx.malloc(want.nbytes + 64)
    try:
        for off in (0, 4, 8):
            for algo in (ft.GEMM_AUTO, ft.GEMM_F4_TC, ft.GEMM_I8_TC, ft.GEMM_POPC_TILED, ft.GEMM_POPC_SIMPLE):
                ctx.fill(d_y, np.full(want.size + 16, np.nan, np.float32))
                ctx.conv(w, d_x, d_t, d_y + off, layer.shape(N), case.alpha, ft.NHWC, ft.PACK_AUTO, algo)
                ctx.sync()
                got = ctx.to_host(d_y, (want.size + 16,), np.float32)
                assert got[off // 4:off // 4 + want.size].tobytes() == want.tobytes(), (off, algo)
                assert np.isnan(got[:off // 4]).all() and np.isnan(got[off // 4 + want.size:]).all(), (off, algo)
    finally:
        for p in (d_t, d_x, d_y):
            ctx.free(p)
        w.free()
