"""GPU parity of the e2m1 convolution (apnn_conv2d_fp4) and of the pooling pass over its rows, against the CPU oracle.
All results are whole numbers: equality."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from gpu_util import spread_bytes, to_dev, to_host
from test_conv_gpu import make_conv

pytestmark = pytest.mark.gpu

CODES = np.array([0, 2, 4, 5], dtype=np.uint8)   # e2m1 codes of the levels 0..3


def spread_nibbles(levels):
    """Levels [..., K] -> e2m1 rows [..., K/2]: nibble i of word q of a 32-element group holds element 31 - (4i + q)."""
    g = CODES[levels].reshape(levels.shape[:-1] + (levels.shape[-1] // 32, 32))[..., ::-1]   # index = bit position
    words = np.zeros(g.shape[:-1] + (4,), dtype=np.uint32)
    for q in range(4):
        for i in range(8):
            words[..., q] |= g[..., 4 * i + q].astype(np.uint32) << (4 * i)
    return words.view(np.uint8).reshape(levels.shape[:-1] + (levels.shape[-1] // 2,))


def expand(planes, signed=False):
    """Device nibble rows of a planes array (cut into 256-element pieces, the last one padded: the expansion is linear)."""
    import apnn_tc_b200 as ap
    flat = planes.reshape(planes.shape[0], -1)
    flat = np.pad(flat, ((0, 0), (0, -flat.shape[1] % 8)))
    return ap.expand_planes_fp4(to_dev(flat.reshape(planes.shape[0], -1, 8)), signed=signed)


def conv_fp4(Wt, X, out, epi, R, CIN, COUT, B, H, Wd, w_signed):
    from apnn_tc_b200 import _cabi
    from apnn_tc_b200.ops import _stream_ptr
    flag = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    x4, w4 = expand(X), expand(Wt, w_signed)
    st = _cabi.lib().apnn_conv2d_fp4(_stream_ptr(), w4.data_ptr(), x4.data_ptr(), out.data_ptr(), B, H, Wd, CIN, COUT, R,
                                     ctypes.byref(epi) if epi is not None else None, flag.data_ptr())
    _cabi.check(st, "apnn_conv2d_fp4")
    assert int(flag.item()) == 0
    return out


SHAPES = [
    # B, H, W, CIN, COUT, R: one tile, ragged channels, half-filled pair, several K blocks, both swizzle spans, wide rows,
    # more tiles than SM pairs
    (1, 2, 2, 128, 32, 3), (2, 7, 7, 512, 512, 3), (3, 13, 13, 384, 384, 3), (1, 56, 56, 256, 256, 3), (2, 5, 100, 128, 64, 3),
    (1, 1, 1, 128, 32, 1), (2, 14, 14, 256, 160, 1), (4, 9, 11, 1152, 288, 1), (24, 28, 28, 128, 512, 3),
    # the widest maps the 256-row box takes: tiles of 64 and of 32 pixels, several waves of them
    (2, 9, 104, 256, 96, 3), (3, 30, 117, 128, 288, 3), (2, 3, 117, 512, 160, 3),
]


@pytest.mark.parametrize("B,H,Wd,CIN,COUT,R", SHAPES)
@pytest.mark.parametrize("wb", [1, 2])
def test_outputs(cuda_device, B, H, Wd, CIN, COUT, R, wb):
    import apnn_tc_b200 as ap
    rng = np.random.default_rng(CIN + COUT + H)
    X, Wt = make_conv(rng, B, H, Wd, CIN, COUT, R, wb, 2)
    v = oracle.conv_popc(Wt, X, threads=8)
    if wb == 1:
        v = oracle.signed_correct(v, oracle.conv_window_sums(X, R), 0)
    args = (R, CIN, COUT, B, H, Wd, wb == 1)
    out = torch.full((B, H, Wd, COUT), -1, dtype=torch.int32, device="cuda")
    assert np.array_equal(to_host(conv_fp4(Wt, X, out, None, *args), np.int32), v)
    T = oracle.fold_bn(rng.uniform(0.5, 1.5, COUT).astype(np.float32), rng.uniform(-1, 1, COUT).astype(np.float32),
                       float(v.mean()), float(v.std()) / 4 + 1, 2)
    T[0] = (-2**31, 0, 2**31 - 1)
    T[1] = T[1][::-1]                      # levels count the thresholds reached, whatever their order
    lv = oracle.levels(v, 2, 2, T)
    epi = ap.make_epilogue("thresholds", 2, thresholds=to_dev(T))
    out = torch.zeros((2, B, H, Wd, COUT // 32), dtype=torch.int32, device="cuda")
    assert np.array_equal(to_host(conv_fp4(Wt, X, out, epi, *args)), oracle.pack_levels(lv, 2))
    halo = 2                               # rows inside a ring that must stay untouched
    for form, width in ((1, COUT), (2, COUT // 2)):
        epi = ap.make_epilogue("thresholds", 2, thresholds=to_dev(T), out_halo=halo)
        epi.out_i8 = form
        out = torch.full((B, H + 2 * halo, Wd + 2 * halo, width), 0xEE, dtype=torch.uint8, device="cuda")
        got = conv_fp4(Wt, X, out, epi, *args).cpu().numpy()
        want = np.full(got.shape, 0xEE, dtype=np.uint8)
        want[:, halo:-halo, halo:-halo] = spread_bytes(lv) if form == 1 else spread_nibbles(lv)
        assert np.array_equal(got, want)
    epi = ap.make_epilogue("thresholds", 1, thresholds=to_dev(T[:, :1].copy()))
    out = torch.zeros((1, B, H, Wd, COUT // 32), dtype=torch.int32, device="cuda")
    assert np.array_equal(to_host(conv_fp4(Wt, X, out, epi, *args)), oracle.requant_pack(v, 1, 2, T[:, :1].copy()))


@pytest.mark.parametrize("widths", [0, 1, 2, 3])
@pytest.mark.parametrize("mode,bits,form", [("thresholds", 2, 2), ("thresholds", 3, 0), ("lowbits", 4, 1), ("lowbits", 2, 2),
                                            ("int32", 0, 0)])
def test_general_epilogue(cuda_device, widths, mode, bits, form):
    """Residuals of either width, wider thresholds, low bits and every output form in the run-time epilogue."""
    import apnn_tc_b200 as ap
    rng = np.random.default_rng(bits * 16 + widths)
    B, H, Wd, CIN, COUT, R = 2, 10, 9, 256, 96, 3
    X, Wt = make_conv(rng, B, H, Wd, CIN, COUT, R, 1, 2)
    v = oracle.signed_correct(oracle.conv_popc(Wt, X, threads=8), oracle.conv_window_sums(X, R), 0)
    res = rng.integers(-3000, 3000, size=(B * H * Wd, COUT)).astype(np.int32)
    v = v + res.reshape(v.shape)
    rin = torch.from_numpy(res.astype(np.int16) if widths & 1 else res).cuda()
    rout = torch.zeros((B * H * Wd, COUT), dtype=torch.int16 if widths & 2 else torch.int32, device="cuda")
    T = np.sort(rng.integers(-4000, 4000, size=(COUT, (1 << bits) - 1)), axis=1).astype(np.int32) if mode == "thresholds" else None
    epi = ap.make_epilogue(mode, bits, thresholds=None if T is None else to_dev(T), residual_in=rin, residual_out=rout,
                           residual_i16=widths)
    epi.out_i8 = form
    if mode == "int32":
        out, want = torch.zeros((B, H, Wd, COUT), dtype=torch.int32, device="cuda"), v
    else:
        lv = oracle.levels(v, bits, 2 if T is not None else 1, T)
        if form:
            out = torch.zeros((B, H, Wd, COUT // form), dtype=torch.uint8, device="cuda")
            want = spread_bytes(lv) if form == 1 else spread_nibbles(lv)
        else:
            out = torch.zeros((bits, B, H, Wd, COUT // 32), dtype=torch.int32, device="cuda")
            want = oracle.pack_levels(lv, bits)
    conv_fp4(Wt, X, out, epi, R, CIN, COUT, B, H, Wd, True)
    got = out.cpu().numpy()
    assert np.array_equal(got.view(want.dtype), want)
    assert np.array_equal(rout.cpu().numpy().astype(np.int32), v.reshape(-1, COUT))


@pytest.mark.parametrize("in_form", [1, 2])
@pytest.mark.parametrize("B,H,Wd,C,ih,oh", [(1, 2, 2, 32, 0, 0), (3, 8, 14, 96, 1, 2), (2, 28, 28, 512, 0, 1)])
def test_pooling_rows(cuda_device, in_form, B, H, Wd, C, ih, oh):
    from apnn_tc_b200 import _cabi
    from apnn_tc_b200.ops import _stream_ptr
    rng = np.random.default_rng(C)
    lv = rng.integers(0, 4, size=(B, H + 2 * ih, Wd + 2 * ih, C), dtype=np.uint32)
    src = torch.from_numpy(spread_bytes(lv) if in_form == 1 else spread_nibbles(lv)).cuda()
    out = torch.full((B, H // 2 + 2 * oh, Wd // 2 + 2 * oh, C // 2), 0xEE, dtype=torch.uint8, device="cuda")
    _cabi.check(_cabi.lib().apnn_maxpool2x2_rows(_stream_ptr(), src.data_ptr(), out.data_ptr(), B, H, Wd, C, ih, oh, in_form, 2))
    inner = lv[:, ih:ih + H, ih:ih + Wd].reshape(B, H // 2, 2, Wd // 2, 2, C).max(axis=(2, 4))
    want = np.full(out.shape, 0xEE, dtype=np.uint8)
    want[:, oh:oh + H // 2, oh:oh + Wd // 2] = spread_nibbles(inner)
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("CIN,COUT,R,stride,mode,res", [(64, 64, 3, 2, "thresholds", False), (128, 288, 1, 2, "lowbits", False),
                                                        (128, 128, 3, 1, "thresholds", True), (256, 256, 3, 1, "thresholds", False)])
def test_int8_layer_writes_nibble_rows(cuda_device, CIN, COUT, R, stride, mode, res):
    """apnn_conv2d_i8_to_fp4: int8 operands in, the next layer's e2m1 operand out, ring untouched."""
    import apnn_tc_b200 as ap
    from apnn_tc_b200 import _cabi
    from apnn_tc_b200.ops import _stream_ptr
    rng = np.random.default_rng(CIN + R)
    B, H, Wd, halo = 3, 14, 18, 1
    p = (R - 1) // 2
    xl = np.zeros((B, H + 2 * p, Wd + 2 * p, CIN), dtype=np.uint32)
    xl[:, p:p + H, p:p + Wd] = rng.integers(0, 4, size=(B, H, Wd, CIN))
    wl = rng.integers(0, 2, size=(COUT, R, R, CIN), dtype=np.uint32)
    X, Wt = oracle.pack_levels(xl, 2), oracle.pack_levels(wl, 1)
    v = oracle.signed_correct(oracle.conv_popc(Wt, X, stride=stride, threads=8), oracle.conv_window_sums(X, R, stride), 0)
    Ho, Wo = v.shape[1:3]
    r = rng.integers(-500, 500, size=v.shape).astype(np.int16)
    if res:
        v = v + r
    T = oracle.fold_bn(np.ones(COUT, np.float32), np.zeros(COUT, np.float32), float(v.mean()), float(v.std()) / 4, 2)
    lv = oracle.levels(v, 2, 2 if mode == "thresholds" else 1, T)
    epi = ap.make_epilogue(mode, 2, thresholds=to_dev(T), out_halo=halo, out_i8=_cabi.ROWS_FP4,
                           residual_in=torch.from_numpy(r).cuda() if res else None, residual_i16=1 if res else 0)
    x8 = torch.from_numpy(spread_bytes(xl)).cuda()
    w8 = torch.from_numpy(spread_bytes((2 * wl.astype(np.int64) - 1).astype(np.uint8).reshape(COUT, -1))).cuda()
    out = torch.full((B, Ho + 2 * halo, Wo + 2 * halo, COUT // 2), 0xEE, dtype=torch.uint8, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    args = (_stream_ptr(), w8.data_ptr(), x8.data_ptr(), out.data_ptr(), B, H, Wd, CIN, COUT, R, stride, 1, ctypes.byref(epi),
            flag.data_ptr())
    assert _cabi.lib().apnn_conv2d_i8(*args) == 1      # nibble rows are this entry point's only
    _cabi.check(_cabi.lib().apnn_conv2d_i8_to_fp4(*args))
    want = np.full(out.shape, 0xEE, dtype=np.uint8)
    want[:, halo:-halo, halo:-halo] = spread_nibbles(lv)
    assert np.array_equal(out.cpu().numpy(), want) and int(flag.item()) == 0


@pytest.mark.parametrize("M,N,K", [(1, 32, 128), (128, 4096, 2304), (64, 512, 9216), (200, 96, 1280), (33, 1000, 4096), (8, 512, 25088),
                                   (2300, 352, 640), (1175, 288, 896), (1024, 1024, 1280), (2240, 1920, 640)])
@pytest.mark.parametrize("sign", ["none", "w", "x"])
def test_gemm_on_narrow_tiles_and_split_k(cuda_device, M, N, K, sign):
    """apnn_linear_fp4 (split K, ragged edges, every output form) and apmm on tcgen05 below the CTA-pair kernel's size."""
    import apnn_tc_b200 as ap
    from apnn_tc_b200 import _cabi
    from apnn_tc_b200.ops import _stream_ptr
    rng = np.random.default_rng(M + N + K)
    wb, xb = (1, 2) if sign == "w" else (2, 1) if sign == "x" else (2, 2)
    W, _ = oracle.value_planes(rng, M, K, wb)
    X, _ = oracle.value_planes(rng, N, K, xb)
    v = oracle.gemm_popc(W, X, threads=8)
    if sign == "w":
        v = oracle.signed_correct(v, oracle.row_sums(X), 1)
    elif sign == "x":
        v = oracle.signed_correct(v, oracle.row_sums(W), 0)
    ws = torch.empty(ap.gemm_workspace_bytes(M, N, K), dtype=torch.uint8, device="cuda")
    epi = ap.make_epilogue("int32", signed=sign)
    assert np.array_equal(to_host(ap.apmm(to_dev(W), to_dev(X), epilogue=epi, algo="tcgen05", workspace=ws), np.int32), v)
    ap.gemm_check(ws, M, N, K)
    T = np.sort(rng.integers(int(v.min()) - 1, int(v.max()) + 2, size=(N, 3)), axis=1).astype(np.int32)
    x4, w4 = expand(W, sign == "w"), expand(X, sign == "x")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")

    def linear(out, e):
        _cabi.check(_cabi.lib().apnn_linear_fp4(_stream_ptr(), x4.data_ptr(), w4.data_ptr(), out.data_ptr(), M, N, K,
                                                ctypes.byref(e), flag.data_ptr()), "apnn_linear_fp4")
        assert int(flag.item()) == 0
        return out
    got = linear(torch.zeros((M, N), dtype=torch.int32, device="cuda"), ap.make_epilogue("int32"))
    assert np.array_equal(to_host(got, np.int32), v)
    sc, bi = rng.uniform(0.5, 1.5, N).astype(np.float32), rng.uniform(-1, 1, N).astype(np.float32)
    e = ap.make_epilogue("float", affine_scale=torch.from_numpy(sc).cuda(), affine_bias=torch.from_numpy(bi).cuda())
    got = linear(torch.zeros((M, N), dtype=torch.float32, device="cuda"), e).cpu().numpy()
    assert np.array_equal(got, oracle.affine_f32(v, sc, bi))
    if N % 32:
        return
    for mode, bits in (("thresholds", 2), ("lowbits", 2), ("lowbits", 5)):
        epi = ap.make_epilogue(mode, bits, signed=sign, thresholds=to_dev(T))
        want = oracle.requant_pack(v, bits, 2 if mode == "thresholds" else 1, T)
        assert np.array_equal(to_host(ap.apmm(to_dev(W), to_dev(X), epilogue=epi, algo="tcgen05", workspace=ws)), want)
    lv = oracle.levels(v, 2, 2, T)
    for form in (1, 2):
        out = linear(torch.zeros((M, N // form), dtype=torch.uint8, device="cuda"),
                     ap.make_epilogue("thresholds", 2, thresholds=to_dev(T), out_i8=form)).cpu().numpy()
        assert np.array_equal(out, spread_bytes(lv) if form == 1 else spread_nibbles(lv))


@pytest.mark.parametrize("H,Wd", [(6, 100), (5, 101), (4, 108), (5, 117), (3, 118)])
@pytest.mark.parametrize("CIN,COUT", [(128, 256), (512, 96)])
def test_wide_maps_from_planes(cuda_device, H, Wd, CIN, COUT):
    """Around the width where packed planes go to int8 instead, and beyond what the 4-bit kernel takes."""
    import apnn_tc_b200 as ap
    rng = np.random.default_rng(Wd)
    X, Wt = make_conv(rng, 2, H, Wd, CIN, COUT, 3, 1, 2)
    v = oracle.conv_popc(Wt, X, threads=8)
    ws = torch.empty(ap.conv_workspace_bytes(2, H, Wd, CIN, COUT, 3), dtype=torch.uint8, device="cuda")
    got = ap.apconv(to_dev(Wt), to_dev(X), algo="tcgen05", workspace=ws)
    assert np.array_equal(to_host(got, np.int32), v)
    v = oracle.signed_correct(v, oracle.conv_window_sums(X, 3), 0)
    T = oracle.fold_bn(np.ones(COUT, np.float32), np.zeros(COUT, np.float32), float(v.mean()), float(v.std()) / 4, 2)
    got = ap.apconv(to_dev(Wt), to_dev(X), algo="tcgen05", workspace=ws, epilogue=ap.make_epilogue("thresholds", 2, signed="w", thresholds=to_dev(T)))
    assert np.array_equal(to_host(got), oracle.requant_pack(v, 2, 2, T))


@pytest.mark.parametrize("B,H,Wd,CIN,COUT,R,stride,mode,pool", [
    (3, 8, 12, 64, 96, 3, 1, "thresholds", "max"), (2, 16, 16, 128, 160, 3, 2, "lowbits", "max"), (2, 12, 8, 128, 64, 1, 1, "thresholds", "avg"),
    (1, 8, 8, 1024, 256, 3, 1, "thresholds", "none"),       # few tiles, 72 K blocks: split K
    (3, 14, 18, 64, 192, 5, 1, "thresholds", "none"), (2, 9, 11, 128, 96, 5, 1, "lowbits", "none"),
    (100, 14, 14, 256, 256, 3, 1, "thresholds", "none"),    # more than one wave of tile pairs: CTA pairs
])
def test_int8_layer_forms_write_nibble_rows(cuda_device, B, H, Wd, CIN, COUT, R, stride, mode, pool):
    """apnn_conv2d_i8_to_fp4 in the forms of the int8 kernel beside the plain one."""
    import apnn_tc_b200 as ap
    from apnn_tc_b200 import _cabi
    from apnn_tc_b200.ops import _stream_ptr
    rng = np.random.default_rng(CIN + R + H)
    p, halo = (R - 1) // 2, 2
    xl = np.zeros((B, H + 2 * p, Wd + 2 * p, CIN), dtype=np.uint32)
    xl[:, p:p + H, p:p + Wd] = rng.integers(0, 4, size=(B, H, Wd, CIN))
    wl = rng.integers(0, 2, size=(COUT, R, R, CIN), dtype=np.uint32)
    X, Wt = oracle.pack_levels(xl, 2), oracle.pack_levels(wl, 1)
    v = oracle.signed_correct(oracle.conv_popc(Wt, X, stride=stride, threads=8), oracle.conv_window_sums(X, R, stride), 0)
    if pool != "none":
        v = oracle.pool2x2(v, 2 if pool == "max" else 1)
    T = oracle.fold_bn(np.ones(COUT, np.float32), np.zeros(COUT, np.float32), float(v.mean()), float(v.std()) / 4, 2)
    want_lv = oracle.levels(v, 2, 2 if mode == "thresholds" else 1, T)
    epi = ap.make_epilogue(mode, 2, thresholds=to_dev(T), out_halo=halo, out_i8=_cabi.ROWS_FP4, pool=pool)
    x8 = torch.from_numpy(spread_bytes(xl)).cuda()
    w8 = torch.from_numpy(spread_bytes((2 * wl.astype(np.int64) - 1).astype(np.uint8).reshape(COUT, -1))).cuda()
    out = torch.full((B, v.shape[1] + 2 * halo, v.shape[2] + 2 * halo, COUT // 2), 0xEE, dtype=torch.uint8, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    _cabi.check(_cabi.lib().apnn_conv2d_i8_to_fp4(_stream_ptr(), w8.data_ptr(), x8.data_ptr(), out.data_ptr(), B, H, Wd, CIN, COUT, R, stride,
                                                  1, ctypes.byref(epi), flag.data_ptr()))
    want = np.full(out.shape, 0xEE, dtype=np.uint8)
    want[:, halo:-halo, halo:-halo] = spread_nibbles(want_lv)
    assert np.array_equal(out.cpu().numpy(), want) and int(flag.item()) == 0
