"""The calls this library is used for, as measurable cases.

Four kinds of work, each through the package's public entry points:

* ``gemm``  -- ``apmm`` on packed planes (weights and activations of a few bits), with and without the fused epilogue;
* ``conv``  -- ``apconv`` on packed NHWC planes with the layer epilogues (thresholds, low bits, 2x2 pooling, int32);
* ``pack``  -- ``images_quantization`` / ``Bit_compression``, the layer-boundary packers;
* ``net``   -- a whole model (``apnn_tc_b200.nets.Network``), called layer by layer or as its captured graph.

Every result is an integer, a packed bit plane, or a float logit made of two separately rounded operations on an exact
integer, so outputs are compared for equality.
"""
import math

import numpy as np
import torch

import apnn_tc_b200 as ap
from apnn_tc_b200 import nets

BATCH_TOP = {"resnet18": 1024, "alexnet": 1024, "vgg_variant": 256}   # largest batch of a drawn network
PAIRS = ((1, 2), (1, 3), (1, 4), (2, 2))                              # weight bits, activation bits
MOST_OPS = 2.0 * 8192 ** 3


def listed():
    return [
        # the smallest call of the reference's published sweep (M = 64, N = K): one launch, all latency
        gemm("gemm_m64_128_w1a2", 1, 2, 64, 128, 128),
        # the largest of that sweep, and the shape its host check uses
        gemm("gemm_m64_1024_w1a2", 1, 2, 64, 1024, 1024),
        # a fully connected layer of AlexNet at batch 128: 9216 -> 4096, +-1 weights, batch norm folded into thresholds
        gemm("fc_128x4096x9216_a2w1", 2, 1, 128, 4096, 9216, out="thresholds", sign="x"),
        # an ordinary ragged problem with an activation width that one e2m1 nibble cannot hold, low bits packed
        gemm("gemm_ragged_w1a4_lowbits", 1, 4, 2300, 2336, 2304, out="lowbits"),
        # the compute-bound square problem, int32 result
        gemm("gemm_8192_w1a2", 1, 2, 8192, 8192, 8192),
        # the reference's single-image convolution with pooling and packing (APConv_w2a2_pack_pool, 16x16)
        conv("conv_b1_16x16_256_w2a2_pool", 2, 2, 1, 16, 256, 256, 3, 1, out="lowbits", pool="avg"),
        # a wide hidden layer at batch 8: +-1 filter, batch norm folded into thresholds, 2-bit packed output
        conv("conv_b8_16x16_1024_w1a2", 1, 2, 8, 16, 1024, 1024, 3, 1, out="thresholds"),
        # feature-map levels to bit planes between two layers
        dict(name="pack_levels_65536x512", kind="pack", source="levels", rows=65536, C=512, bits=2),
        # whole networks: a single small request through forward(), the multi-GPU share, a full batch, the wide model
        net("resnet18_b8", "resnet18", 8, graph=False),
        net("alexnet_b128_graph", "alexnet", 128, graph=True),
        net("resnet18_b1024_graph", "resnet18", 1024, graph=True),
        net("vgg_variant_b128_graph", "vgg_variant", 128, graph=True),
    ]


def gemm(name, wbits, xbits, M, N, K, out="int32", sign="none"):
    return dict(name=name, kind="gemm", wbits=wbits, xbits=xbits, M=M, N=N, K=K, out=out, sign=sign)


def conv(name, wbits, xbits, B, H, C, O, R, stride, out="int32", pool="none"):
    return dict(name=name, kind="conv", wbits=wbits, xbits=xbits, B=B, H=H, C=C, O=O, R=R, stride=stride, out=out, pool=pool)


def net(name, model, batch, graph):
    return dict(name=name, kind="net", model=model, batch=batch, graph=graph)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("gemm", "gemm", "conv", "pack", "net"))
    if kind == "gemm":
        small = rng.random() < 0.4
        wbits, xbits = rng.choice(PAIRS)
        out = rng.choice(("int32", "int32", "lowbits", "thresholds"))
        if small:     # the launch-bound sweep and its neighbourhood
            M, N, K = rng.choice((64, rng.randint(1, 256))), _log(rng, 32, 1024), 128 * rng.randint(1, 8)
        else:
            M, N, K = _log(rng, 64, 8192), _log(rng, 64, 8192), 128 * _log(rng, 2, 72)
        if out != "int32":
            N = (N + 31) // 32 * 32
        sign = "w" if wbits == 1 and out == "thresholds" else "none"
        if out == "thresholds" and rng.random() < 0.4:    # a fully connected layer: activations first, +-1 weights second
            wbits, xbits, sign = 2, 1, "x"
        c = gemm("", wbits, xbits, M, N, K, out, sign)
    elif kind == "conv":
        wbits, xbits = rng.choice(PAIRS)
        pool = rng.choice(("none", "none", "none", "avg", "max"))
        R = rng.choice((1, 3, 3, 3, 5))
        stride = rng.choice((1, 1, 1, 2))
        H = _log(rng, 7, 56)
        if pool != "none":
            H = max(8, H // 4 * 4)      # the output extent has to be even
        C, O = 128 * rng.randint(1, 8), 32 * _log(rng, 2, 32)
        B = _log(rng, 1, 32)
        while 2.0 * B * H * H * C * O * R * R > MOST_OPS / 4:
            B = max(1, B // 2)
            if B == 1:
                H = max(8, H // 8 * 4)
        out = rng.choice(("int32", "lowbits", "thresholds", "thresholds"))
        c = conv("", wbits, xbits, B, H, C, O, R, stride, out, pool)
    elif kind == "pack":
        C = rng.choice((3, rng.randint(1, 64), 64 * rng.randint(1, 16), rng.randint(65, 1024)))
        rows = max(64, _log(rng, 1024, 1 << 20) * 32 // max(C, 32))
        c = dict(kind="pack", source=rng.choice(("levels", "float")), rows=rows, C=C, bits=rng.choice((1, 2, 2, 3, 4)))
    else:
        model = rng.choice(sorted(nets.MODELS))
        c = net("", model, _log(rng, 1, BATCH_TOP[model]), graph=rng.random() < 0.6)
    c.pop("name", None)
    return c


# ----------------------------------------------------------------------------- inputs
def _words(gen, shape):
    """Uniform bits, 32 per word: uniform levels in their bit planes."""
    return torch.randint(-2 ** 31, 2 ** 31, shape, dtype=torch.int64, device="cuda", generator=gen).to(torch.int32)


def _thresholds(seed, channels, fan_in, wbits, xbits, signed):
    """Batch norm (scale U[0.5, 1.5], bias U[-1, 1]) folded into the 2-bit quantiser's thresholds, centred on the values
    that uniform operands give, so that every level occurs."""
    rng = np.random.default_rng(seed)
    lv = np.arange(1 << xbits, dtype=np.float64)
    wv = np.array([-1.0, 1.0]) if signed else np.arange(1 << wbits, dtype=np.float64)
    mean = lv.mean() * wv.mean()
    var = (lv ** 2).mean() * (wv ** 2).mean() - mean ** 2
    T = nets.fold_thresholds(rng.uniform(0.5, 1.5, channels).astype(np.float32), rng.uniform(-1, 1, channels).astype(np.float32),
                             fan_in * mean, math.sqrt(var * fan_in) / 4, 2)
    return torch.from_numpy(T).cuda()


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "gemm":
        M, N, K, wb, xb = case["M"], case["N"], case["K"], case["wbits"], case["xbits"]
        s.W = _words(gen, (wb, M, K // 32))
        s.X = _words(gen, (xb, N, K // 32))
        s.epi = None
        if case["out"] == "int32":
            s.D = torch.empty((M, N), dtype=torch.int32, device="cuda")
        else:
            bits = 2
            s.D = torch.empty((bits, M, N // 32), dtype=torch.int32, device="cuda")
            if case["out"] == "lowbits":
                s.epi = ap.make_epilogue("lowbits", bits, signed=case["sign"])
            else:
                # the signed operand is the one-bit one; the other holds the levels
                first_is_level = case["sign"] == "x"
                s.T = _thresholds(seed, N, K, xb if first_is_level else wb, wb if first_is_level else xb, case["sign"] != "none")
                s.epi = ap.make_epilogue("thresholds", bits, signed=case["sign"], thresholds=s.T)
        s.ws = torch.empty(ap.gemm_workspace_bytes(M, N, K, wb, xb), dtype=torch.uint8, device="cuda")
    elif kind == "conv":
        B, H, C, O, R, st, wb, xb = (case[k] for k in ("B", "H", "C", "O", "R", "stride", "wbits", "xbits"))
        p = (R - 1) // 2
        s.X = _words(gen, (xb, B, H + 2 * p, H + 2 * p, C // 32))
        if p:                      # the stored halo is padding
            s.X[:, :, :p] = 0
            s.X[:, :, -p:] = 0
            s.X[:, :, :, :p] = 0
            s.X[:, :, :, -p:] = 0
        s.W = _words(gen, (wb, O, R, R, C // 32))
        signed = wb == 1 and case["out"] == "thresholds"
        T = _thresholds(seed, O, R * R * C, wb, xb, signed) if case["out"] == "thresholds" else None
        s.epi = ap.make_epilogue(case["out"], 0 if case["out"] == "int32" else 2, signed="w" if signed else "none",
                                 pool=case["pool"], thresholds=T)
        Ho = (H - 1) // st + 1
        if case["pool"] != "none":
            Ho //= 2
        s.D = torch.empty((B, Ho, Ho, O) if case["out"] == "int32" else (2, B, Ho, Ho, O // 32), dtype=torch.int32, device="cuda")
        s.ws = torch.empty(ap.conv_workspace_bytes(B, H, H, C, O, R), dtype=torch.uint8, device="cuda")
    elif kind == "pack":
        shape, bits = (case["rows"], case["C"]), case["bits"]
        if case["source"] == "levels":
            s.X = torch.randint(0, 1 << bits, shape, dtype=torch.int32, device="cuda", generator=gen)
        else:
            s.X = torch.rand(shape, device="cuda", generator=gen) * 20.0 - 10.0
        s.D = torch.empty((bits, case["rows"], (case["C"] + 127) // 128 * 4), dtype=torch.int32, device="cuda")
    else:
        spec = nets.MODELS[case["model"]]()
        s.net = nets.Network(spec, case["batch"], nets.make_params(spec, seed=seed))
        s.images = torch.rand((case["batch"], spec.image_hw, spec.image_hw, spec.image_channels), device="cuda",
                              generator=gen) * 20.0 - 10.0
        if case["graph"]:
            s.net.capture(s.images)
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "gemm":
        return ap.apmm(s.W, s.X, s.D, epilogue=s.epi, workspace=s.ws)
    if kind == "conv":
        return ap.apconv(s.W, s.X, s.D, stride=case["stride"], epilogue=s.epi, algo="auto", workspace=s.ws)
    if kind == "pack":
        pack = ap.Bit_compression if case["source"] == "levels" else ap.images_quantization
        return pack(s.X, case["bits"], s.D)
    return s.net.replay() if case["graph"] else s.net.forward(s.images)


def work(case):
    kind = case["kind"]
    if kind == "gemm":
        M, N, K = case["M"], case["N"], case["K"]
        out = 4 * M * N if case["out"] == "int32" else 2 * M * N // 8
        thr = 12 * N if case["out"] == "thresholds" else 0
        return {"bytes": (case["wbits"] * M + case["xbits"] * N) * K // 8 + out + thr, "flops": 2.0 * M * N * K}
    if kind == "conv":
        B, H, C, O, R = (case[k] for k in ("B", "H", "C", "O", "R"))
        Ho = (H - 1) // case["stride"] + 1
        outs = B * (Ho // 2) ** 2 * O if case["pool"] != "none" else B * Ho * Ho * O
        b = case["xbits"] * B * (H + R - 1) ** 2 * C // 8 + case["wbits"] * O * R * R * C // 8
        b += 4 * outs if case["out"] == "int32" else 2 * outs // 8
        return {"bytes": b + (12 * O if case["out"] == "thresholds" else 0), "flops": 2.0 * B * Ho * Ho * O * R * R * C}
    if kind == "pack":
        rows, C = case["rows"], case["C"]
        return {"bytes": 4 * rows * C + case["bits"] * rows * ((C + 127) // 128 * 128) // 8, "flops": 0}
    spec = nets.MODELS[case["model"]]()
    macs, weights = _net_macs(spec)
    B = case["batch"]
    image = 4 * spec.image_hw ** 2 * spec.image_channels
    return {"bytes": B * image + weights // 8 + 4 * B * spec.layers[-1].cout, "flops": 2.0 * B * macs}


def _net_macs(spec):
    """Multiply-adds of one image and one-bit weights of a model list (the shape rules of nets.make_params)."""
    dims, prev, macs, weights = {}, None, 0, 0
    for ls in spec.layers:
        src = ls.src or prev
        if ls.kind == "conv":
            H, W, C = dims[src] if src else (spec.image_hw, spec.image_hw, spec.image_channels)
            Ho, Wo = (H - 1) // ls.stride + 1, (W - 1) // ls.stride + 1
            k = ls.R * ls.R * ls.cin
            macs += Ho * Wo * k * ls.cout
            dims[ls.name] = (Ho // ls.pool, Wo // ls.pool, ls.cout)
        else:
            k = ls.cin or dims[src][0] * dims[src][1] * dims[src][2]
            macs += k * ls.cout
            dims[ls.name] = (1, 1, ls.cout)
        weights += k * ls.cout
        prev = ls.name
    return macs, weights


def tolerance(case):
    return "exact"
