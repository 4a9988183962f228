"""The work this framework is used for, as measurable cases over its public entry points.

A case is one of five kinds:

  layer    one device-resident convolution or fully connected layer (``Context.conv``)
  chain    a network of layers on the device (``ConvStack`` with 4-bit images between the layers)
  packed   the reference's two steps by themselves on the device: quantise + im2row into the packed
           matrix, then the packed GEMM (``Context.pack``, ``Context.gemm``)
  drop_in  one layer through the reference's own call, pageable host memory in and out (``tnns_conv``)
  host     one layer over page-locked host buffers, sliced and overlapped (``Context.conv_host``)

Every result is an integer sum under an exact PReLU slope, so all outputs are compared bit for bit.
Sizes come from the benchmark configurations and the reference's shape tables (``fastertnn_b200.workloads``).
"""
import math

import numpy as np
import torch

import fastertnn_b200 as ft
from fastertnn_b200.stack import ConvStack
from fastertnn_b200.workloads import RESNET18_STACK, Layer, model_layers

ALPHA = 0.5
TYPES = {"tnn": ft.TNN, "tbn": ft.TBN, "btn": ft.BTN, "bnn": ft.BNN}
_CONTEXT = None


def _context():
    """A program has one context per host thread."""
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = ft.Context(0)
    return _CONTEXT


def _layer_case(name, kind, type_, N, C, H, W, KN, KH, KW, P, S, layout="nchw"):
    case = {"kind": kind, "type": type_, "N": N, "C": C, "H": H, "W": W, "KN": KN, "KH": KH, "KW": KW, "P": P, "S": S, "layout": layout}
    return dict(case, name=name) if name else case


def listed():
    return [
        # The first shape of the reference's own run: the smallest calls, where launches and the host path count.
        _layer_case("small_layer_b8", "layer", "tnn", 8, 32, 7, 7, 32, 3, 3, 0, 1),
        # One image through a middle layer of an image network: what an interactive service asks for.
        _layer_case("conv56_b1_tbn", "layer", "tbn", 1, 256, 56, 56, 256, 3, 3, 1, 1),
        # A downsampling layer with binary activations.
        _layer_case("down14_b8_btn", "layer", "btn", 8, 256, 14, 14, 256, 3, 3, 1, 2),
        # Channel counts and image sizes that are no multiple of anything (a shape of the reference's run).
        _layer_case("ragged_b8", "layer", "tnn", 8, 320, 15, 23, 320, 3, 3, 1, 2),
        # A fully connected layer: M = 1024, K = 4096, N = 1024.
        _layer_case("fc_1024", "layer", "tnn", 1024, 4096, 1, 1, 1024, 1, 1, 0, 1),
        # The slice of the large layer that one of eight GPUs owns, pixel-major.
        _layer_case("large_b8_nhwc", "layer", "tnn", 8, 512, 32, 32, 512, 3, 3, 1, 1, "nhwc"),
        # The large layer on one GPU (the benchmark's default).
        _layer_case("large_b64", "layer", "tnn", 64, 512, 32, 32, 512, 3, 3, 1, 1),
        # An 11-layer stack at batch 256: offline throughput of a whole network.
        {"name": "stack_b256", "kind": "chain", "type": "tnn", "net": "stack", "N": 256},
        # A whole network from its three-channel entry layer on, at the batch the reference's driver uses.
        {"name": "resnet18_b8", "kind": "chain", "type": "tnn", "net": "resnet18", "N": 8},
        # The packed matrix and the packed GEMM, for programs that keep the reference's two steps.
        _layer_case("packed_large_b8", "packed", "tnn", 8, 512, 32, 32, 512, 3, 3, 1, 1),
        # The reference's call on the reference's buffers: a shape of its run at its batch.
        _layer_case("drop_in_b8", "drop_in", "tnn", 8, 256, 14, 14, 256, 3, 3, 1, 2),
        # The large layer end to end from host memory.
        _layer_case("host_large_b64", "host", "tnn", 64, 512, 32, 32, 512, 3, 3, 1, 1),
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# floats in and out and operations of a layer, per kind: the largest listed case of that kind
_MOST = {"layer": (67.2e6, 310e9), "packed": (8.4e6, 39e9), "drop_in": (6e6, 20e9), "host": (67.2e6, 310e9)}


def draw(rng):
    kind = rng.choices(["layer", "chain", "packed", "drop_in", "host"], [12, 3, 2, 2, 1])[0]
    if kind == "chain":
        net = rng.choice(["stack", "resnet18"])
        return {"kind": "chain", "type": rng.choice(["tnn", "tnn", "tbn"]), "net": net, "N": _log(rng, 1, 256 if net == "stack" else 24)}
    floats, ops = _MOST[kind]
    while True:
        type_ = rng.choices(["tnn", "tbn", "btn", "bnn"], [5, 2, 2, 1])[0]
        layout = rng.choice(["nchw", "nhwc"]) if kind in ("layer", "host") else "nchw"
        KH, KW, P, S = rng.choices([(3, 3, 1, 1), (3, 3, 1, 2), (1, 1, 0, 1), (1, 1, 0, 2), (5, 5, 2, 1), (5, 3, 1, 2), (3, 3, 0, 1)], [8, 4, 3, 1, 1, 1, 1])[0]
        C, KN = (rng.choice([32, 64, 96, 128, 192, 256, 320, 384, 512, 1024]) if rng.random() < 0.7 else _log(rng, 17, 1100) for _ in range(2))
        H = _log(rng, 7, 112)
        W = H if rng.random() < 0.7 else _log(rng, 7, 112)
        N = _log(rng, 1, 256)
        shape = rng.random()
        if shape < 0.08:      # an image network's entry layer
            C, (KH, KW, P, S), H, W, KN = 3, rng.choice([(7, 7, 3, 2), (3, 3, 1, 1), (3, 3, 1, 2)]), 224, 224, rng.choice([32, 64, 96])
        elif shape < 0.18:    # a fully connected layer
            H = W = KH = KW = S = 1
            P, C, KN, N = 0, _log(rng, 256, 8192), _log(rng, 10, 4096), _log(rng, 1, 4096)
        case = _layer_case(None, kind, type_, N, C, H, W, KN, KH, KW, P, S, layout)
        L = _geometry(case)
        if N * (C * H * W + KN * L.OH * L.OW) <= floats and 1e6 <= L.ops(N) <= ops:
            return case


def _geometry(case):
    return Layer(case["C"], case["H"], case["W"], case["KN"], case["KH"], case["KW"], case["P"], case["S"])


def _network(case):
    return RESNET18_STACK if case["net"] == "stack" else model_layers("resnet18")


# ---- inputs ----------------------------------------------------------------------------------------

def _activations(case, C, H, W, g):
    """fp32 activations uniform in [-1, 1) and one threshold per image, near 0.25 (ternary) or 0 (binary)."""
    N = case["N"]
    x = torch.empty((N, H, W, C) if case.get("layout") == "nhwc" else (N, C, H, W), device="cuda").uniform_(-1, 1, generator=g)
    t = torch.empty(N, device="cuda").uniform_(-0.05, 0.05, generator=g)
    return x, (t + 0.25 if TYPES[case["type"]] in (ft.TNN, ft.TBN) else t)


def _packed_weights(case, L, g):
    """Weights i.i.d. uniform in {-1, 0, +1} or {-1, +1}, packed as the reference packs them, on the host."""
    ternary = TYPES[case["type"]] in (ft.TNN, ft.BTN)
    shape = (L.KN, L.C, L.KH, L.KW)
    w = torch.randint(-1, 2, shape, device="cuda", generator=g).float() if ternary else torch.randint(0, 2, shape, device="cuda", generator=g).float() * 2 - 1
    thr = torch.full((L.KN,), 0.5 if ternary else 0.0, device="cuda")
    packed = torch.empty((L.KN, (2 if ternary else 1) * ft.k_padded(L.C, L.KH, L.KW)), dtype=torch.int64, device="cuda")
    _context().pack_weights_device(ternary, w.data_ptr(), thr.data_ptr(), packed.data_ptr(), L.KN, L.C, L.KH, L.KW)
    return packed.cpu().numpy()


class _Owned:
    """Releases one of the library's handles with the last reference to it."""

    def __init__(self, handle, release):
        self.handle, self.release = handle, release

    def __del__(self):
        self.release()


class _ChainBuffer:
    """The chain's input or output buffer, for torch; a tensor made of it keeps the chain alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": tuple(shape), "typestr": "<f4", "version": 2}

    def tensor(self):
        return torch.as_tensor(self, device="cuda")


class _State:
    """What a program holds for one case."""

    def __init__(self, case):
        self.case, self.kind, self.type = case, case["kind"], TYPES[case["type"]]
        self.layout = ft.NHWC if case.get("layout") == "nhwc" else ft.NCHW

    def own(self, handle, release):
        self.owned, self.handle = _Owned(handle, release), handle


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    s = _State(case)
    ctx = _context()
    if s.kind == "chain":
        layers = _network(case)
        chain = ConvStack(ctx, s.type, layers, [_packed_weights(case, L, g) for L in layers], case["N"], 0.25, ALPHA, ft.NCHW, chain="image")
        s.own(chain, chain.close)
        first, last = layers[0], layers[-1]
        x, _ = _activations(case, first.C, first.H, first.W, g)
        _ChainBuffer(s.owned, chain.input_ptr(), x.shape).tensor().copy_(x)  # where the chain reads its input
        s.y = _ChainBuffer(s.owned, chain.output_ptr(), (case["N"], last.KN, last.OH, last.OW)).tensor()
        return s
    L = _geometry(case)
    s.L, s.shape = L, L.shape(case["N"])
    packed = _packed_weights(case, L, g)
    s.x, s.thr = _activations(case, L.C, L.H, L.W, g)
    if s.kind == "drop_in":
        s.x, s.thr, s.packed = s.x.cpu().numpy(), s.thr.cpu().numpy(), packed
        return s
    w = ctx.upload_weights(s.type, packed, L.C, L.KH, L.KW)
    s.own(w, w.free)
    y_shape = (case["N"], L.OH, L.OW, L.KN) if s.layout == ft.NHWC else (case["N"], L.KN, L.OH, L.OW)
    if s.kind == "host":
        s.x, s.thr = s.x.cpu().pin_memory(), s.thr.cpu().pin_memory()
        s.y = torch.empty(y_shape, pin_memory=True)
        return s
    s.y = torch.empty(y_shape, device="cuda")
    if s.kind == "packed":
        planes = 2 if s.type in (ft.TNN, ft.TBN) else 1
        s.a = torch.empty((case["N"] * L.OH * L.OW, planes * ft.k_padded(L.C, L.KH, L.KW)), dtype=torch.int64, device="cuda")
    return s


def run(s):
    ctx = _CONTEXT
    if s.kind == "layer":
        ctx.conv(s.handle, s.x.data_ptr(), s.thr.data_ptr(), s.y.data_ptr(), s.shape, ALPHA, s.layout)
        return s.y
    if s.kind == "chain":
        s.handle.run()
        return s.y
    L = s.L
    if s.kind == "packed":
        ctx.pack(s.type in (ft.TNN, ft.TBN), s.x.data_ptr(), s.thr.data_ptr(), s.a.data_ptr(), s.shape)
        ctx.gemm(s.handle, s.a.data_ptr(), s.y.data_ptr(), s.case["N"], L.OH, L.OW, ALPHA)
        return s.a, s.y
    if s.kind == "host":
        ctx.conv_host(s.handle, s.x.data_ptr(), s.thr.data_ptr(), s.y.data_ptr(), s.shape, ALPHA, s.layout)
        return s.y
    return ft.tnns_conv(s.type, s.x, s.thr, s.packed, (L.KH, L.KW), (L.P, L.P), (L.S, L.S), ALPHA)


def work(case):
    """The fp32 input and the weight bits read, the fp32 output (and the packed matrix) written, 2*M*N*K operations."""
    N, type_ = case["N"], TYPES[case["type"]]
    layers = _network(case) if case["kind"] == "chain" else [_geometry(case)]
    first, last = layers[0], layers[-1]
    planes = 2 if type_ in (ft.TNN, ft.BTN) else 1
    b = 4 * N * (first.C * first.H * first.W + 1) + 4 * N * last.KN * last.OH * last.OW + sum(planes * L.KN * L.C * L.KH * L.KW // 8 for L in layers)
    if case["kind"] == "packed":
        b += N * last.OH * last.OW * ft.k_padded(last.C, last.KH, last.KW) * 8 * (2 if type_ in (ft.TNN, ft.TBN) else 1)
    return {"bytes": b, "flops": sum(L.ops(N) for L in layers)}


def tolerance(case):
    """Integer sums below 2^22 times a power of two: the same bits from every correct implementation."""
    return "exact"
