"""The e2m1 kernels hold sums in fp32 and are taken while no sum reaches 2^24.  Here the sums come as close to that as the
checks admit: levels 3 except for one element in a thousand, so partial sums of every size up to the limit occur with all their
low bits, in one accumulator and split over a cluster.  Whole numbers: equality with a float64 product."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from gpu_util import to_dev, to_host
from test_conv_fp4_gpu import expand

pytestmark = pytest.mark.gpu

LIMIT = 2 ** 24
K_MAX = (LIMIT - 1) // 9 // 128 * 128          # 9 * K < 2^24, K a multiple of 128


def near_max(rng, shape, bits):
    """Levels of `bits` bits, all at their maximum but one in a thousand."""
    top = (1 << bits) - 1
    lv = np.full(shape, top, dtype=np.uint32)
    flat = lv.reshape(-1)
    at = rng.integers(0, flat.size, size=max(1, flat.size // 1000))
    flat[at] = rng.integers(0, top, size=at.size)
    return lv


def product(wl, xl):
    """wl [M, K] @ xl [N, K]^T in float64 (exact: the sums stay below 2^53), in pieces of K."""
    out = torch.zeros((wl.shape[0], xl.shape[0]), dtype=torch.float64, device="cuda")
    for k in range(0, wl.shape[1], 1 << 17):
        w, x = (torch.from_numpy(a[:, k:k + (1 << 17)].astype(np.float64)).cuda() for a in (wl, xl))
        out += w @ x.T
    return out.cpu().numpy().astype(np.int64)


@pytest.mark.parametrize("kernel", ["planes", "linear", "pair"])
@pytest.mark.parametrize("wb,xb,signed,M,N", [(2, 2, False, 33, 64), (1, 2, True, 70, 32)])
def test_gemm_sums_just_below_the_limit(cuda_device, kernel, wb, xb, signed, M, N):
    import apnn_tc_b200 as ap
    from apnn_tc_b200 import _cabi
    from apnn_tc_b200.ops import _stream_ptr
    K = K_MAX if kernel != "pair" else K_MAX // 256 * 256
    rng = np.random.default_rng(K + M)
    wl, xl = near_max(rng, (M, K), wb), near_max(rng, (N, K), xb)
    if signed:
        wl[::2] = 1 - wl[::2]                  # rows of almost only -1 beside rows of almost only +1
    W, X = oracle.pack_levels(wl, wb), oracle.pack_levels(xl, xb)
    want = product(2.0 * wl - 1.0 if signed else wl, xl)
    assert np.abs(want).max() > (0.99 * 3 * K if signed else 0.99 * LIMIT) and np.abs(want).max() < LIMIT
    L, flag = _cabi.lib(), torch.full((1,), 7, dtype=torch.int32, device="cuda")
    T = np.stack([want[0], want[0] + 1, want[0] + 2], axis=1).astype(np.int32)     # decided by the lowest bit
    packed = want[:, :, None] >= T[None]
    if kernel == "planes":
        Wd, Xd = to_dev(W), to_dev(X)

        def call(out, e):
            e.signed_operand = _cabi.SIGN_W if signed else _cabi.SIGN_NONE
            return L.apnn_gemm_planes(_stream_ptr(), wb, xb, Wd.data_ptr(), Xd.data_ptr(), out.data_ptr(), M, N, K, ctypes.byref(e), flag.data_ptr())
    else:
        W4, X4 = expand(W, signed), expand(X)
        fn = L.apnn_linear_fp4 if kernel == "linear" else L.apnn_gemm_fp4

        def call(out, e):
            return fn(_stream_ptr(), W4.data_ptr(), X4.data_ptr(), out.data_ptr(), M, N, K, ctypes.byref(e), flag.data_ptr())
    out = torch.full((M, N), -1, dtype=torch.int32, device="cuda")
    _cabi.check(call(out, ap.make_epilogue("int32")))
    assert int(flag.item()) == 0 and np.array_equal(to_host(out, np.int32), want)
    out = torch.zeros((2, M, N // 32), dtype=torch.int32, device="cuda")
    _cabi.check(call(out, ap.make_epilogue("thresholds", 2, thresholds=to_dev(T))))
    assert int(flag.item()) == 0 and np.array_equal(to_host(out), oracle.pack_levels(packed.sum(axis=2).astype(np.uint32), 2))


@pytest.mark.parametrize("residual", [False, True])
def test_convolution_sums_just_below_the_limit(cuda_device, residual):
    """3x3, int32 rows and thresholds one apart; with int16 residuals added as floats the sum still has to stay below 2^24."""
    import apnn_tc_b200 as ap
    from apnn_tc_b200 import _cabi
    from apnn_tc_b200.ops import _stream_ptr
    CIN, COUT, H = ((LIMIT - 1 - (32768 if residual else 0)) // 81) // 128 * 128, 32, 3
    rng = np.random.default_rng(CIN)
    xl, wl = np.zeros((1, H + 2, H + 2, CIN), dtype=np.uint32), near_max(rng, (COUT, 3, 3, CIN), 2)
    xl[:, 1:-1, 1:-1] = near_max(rng, (1, H, H, CIN), 2)
    windows = np.stack([xl[0, h:h + 3, w:w + 3].reshape(-1) for h in range(H) for w in range(H)])
    v = product(windows, wl.reshape(COUT, -1))
    assert v.max() > 0.99 * 81 * CIN
    res = rng.integers(32700, 32768, size=v.shape).astype(np.int16) if residual else np.zeros(v.shape, np.int16)
    rin, rout = torch.from_numpy(res).cuda(), torch.zeros(v.shape, dtype=torch.int16, device="cuda")
    v = v + res
    assert v.max() < LIMIT
    centre = v[4]
    T = np.stack([centre, centre + 1, centre + 2], axis=1).astype(np.int32)
    x4, w4 = expand(oracle.pack_levels(xl, 2)), expand(oracle.pack_levels(wl, 2))
    flag = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    extra = dict(residual_in=rin, residual_out=rout, residual_i16=3) if residual else {}
    for mode, bits in (("thresholds", 2), ("int32", 0)):
        epi = ap.make_epilogue(mode, bits, thresholds=to_dev(T), **extra)
        out = torch.zeros((2, H * H, 1) if bits else (H * H, COUT), dtype=torch.int32, device="cuda")
        _cabi.check(_cabi.lib().apnn_conv2d_fp4(_stream_ptr(), w4.data_ptr(), x4.data_ptr(), out.data_ptr(), 1, H, H, CIN, COUT, 3,
                                                ctypes.byref(epi), flag.data_ptr()))
        assert int(flag.item()) == 0
        if bits:
            levels = (v[:, :, None] >= T[None]).sum(axis=2).astype(np.uint32)
            assert np.array_equal(to_host(out), oracle.pack_levels(levels, 2))
        else:
            assert np.array_equal(to_host(out, np.int32), v)
        if residual:
            assert np.array_equal(rout.cpu().numpy(), np.clip(v, -32768, 32767))
