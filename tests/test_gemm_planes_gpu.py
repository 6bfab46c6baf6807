"""GPU parity of the one-launch GEMM from packed planes (apnn_gemm_planes) against the CPU oracle: whole numbers, equality."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu

# one piece of K, half a K block at the end, partial tiles in both directions, widths of the pixel tile, split K over
# clusters of 2, 4 and 8, several waves
SHAPES = [(1, 1, 128), (31, 33, 384), (64, 128, 128), (100, 96, 640), (129, 257, 1024), (224, 512, 2048), (64, 1024, 8192),
          (128, 4096, 9216), (64, 128, 16384), (700, 416, 1152), (2048, 1056, 256), (512, 512, 4096), (300, 2304, 6144), (2100, 1700, 1024)]


def run(W, X, out, epi, wb, xb, M, N, K):
    from apnn_tc_b200 import _cabi
    from apnn_tc_b200.ops import _stream_ptr
    flag = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    _cabi.check(_cabi.lib().apnn_gemm_planes(_stream_ptr(), wb, xb, W.data_ptr(), X.data_ptr(), out.data_ptr(), M, N, K,
                                             ctypes.byref(epi), flag.data_ptr()), "apnn_gemm_planes")
    assert int(flag.item()) == 0
    return out


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("wb,xb,sign", [(1, 2, "none"), (1, 2, "w"), (2, 1, "x"), (2, 2, "none"), (1, 1, "w")])
def test_planes_gemm(cuda_device, M, N, K, wb, xb, sign):
    import apnn_tc_b200 as ap
    rng = np.random.default_rng(M * 7 + N + K)
    W, _ = oracle.value_planes(rng, M, K, wb)
    X, _ = oracle.value_planes(rng, N, K, xb)
    v = oracle.gemm_popc(W, X, threads=8)
    if sign == "w":
        v = oracle.signed_correct(v, oracle.row_sums(X), 1)
    elif sign == "x":
        v = oracle.signed_correct(v, oracle.row_sums(W), 0)
    Wd, Xd = to_dev(W), to_dev(X)
    out = torch.full((M, N), -1, dtype=torch.int32, device="cuda")
    assert np.array_equal(to_host(run(Wd, Xd, out, ap.make_epilogue("int32", signed=sign), wb, xb, M, N, K), np.int32), v)
    if N % 32:
        return
    T = np.sort(rng.integers(int(v.min()) - 1, int(v.max()) + 2, size=(N, 3)), axis=1).astype(np.int32)
    for mode, bits in (("thresholds", 2), ("lowbits", 2), ("lowbits", 4)):
        epi = ap.make_epilogue(mode, bits, signed=sign, thresholds=to_dev(T))
        out = torch.zeros((bits, M, N // 32), dtype=torch.int32, device="cuda")
        want = oracle.requant_pack(v, bits, 2 if mode == "thresholds" else 1, T)
        assert np.array_equal(to_host(run(Wd, Xd, out, epi, wb, xb, M, N, K)), want)


def test_planes_gemm_residuals_and_large_thresholds(cuda_device):
    import apnn_tc_b200 as ap
    M, N, K = 130, 96, 1152
    rng = np.random.default_rng(5)
    W, _ = oracle.value_planes(rng, M, K, 1)
    X, _ = oracle.value_planes(rng, N, K, 2)
    res = rng.integers(-2**31, 2**31 - 1, size=(M, N), dtype=np.int64).astype(np.int32)
    v = (oracle.gemm_popc(W, X, threads=8).astype(np.int64) + res).astype(np.int32)
    T = np.sort(rng.integers(-2**31, 2**31 - 1, size=(N, 3)), axis=1).astype(np.int32)
    rout = torch.zeros((M, N), dtype=torch.int32, device="cuda")
    epi = ap.make_epilogue("thresholds", 2, thresholds=to_dev(T), residual_in=to_dev(res), residual_out=rout)
    out = torch.zeros((2, M, N // 32), dtype=torch.int32, device="cuda")
    assert np.array_equal(to_host(run(to_dev(W), to_dev(X), out, epi, 1, 2, M, N, K)), oracle.requant_pack(v, 2, 2, T))
    assert np.array_equal(rout.cpu().numpy(), v)


@pytest.mark.parametrize("offset", [0, 4, 16, 1, 18])
@pytest.mark.parametrize("M,N,K,mode", [(64, 128, 128, "int32"), (64, 128, 128, "lowbits"), (1024, 1024, 1024, "int32")])
def test_automatic_choice_with_a_workspace_at_any_offset(cuda_device, offset, M, N, K, mode):
    """The status flag is left at 0 wherever the workspace lies, by the kernel or, at an odd address, by a memset."""
    import apnn_tc_b200 as ap
    from apnn_tc_b200 import _cabi
    from apnn_tc_b200.ops import _stream_ptr
    rng = np.random.default_rng(offset + M)
    W, _ = oracle.value_planes(rng, M, K, 1)
    X, _ = oracle.value_planes(rng, N, K, 2)
    v = oracle.gemm_popc(W, X, threads=8)
    size = ap.gemm_workspace_bytes(M, N, K)
    ws = torch.full((size + 32,), 0xEE, dtype=torch.uint8, device="cuda")[offset:offset + size]
    epi = ap.make_epilogue(mode, 2) if mode != "int32" else None
    got = ap.apmm(to_dev(W), to_dev(X), workspace=ws, epilogue=epi)
    _cabi.check(_cabi.lib().apnn_gemm_check(_stream_ptr(), ws.data_ptr(), M, N, K))
    if mode == "int32":
        assert np.array_equal(to_host(got, np.int32), v)
    else:
        assert np.array_equal(to_host(got), oracle.requant_pack(v, 2, 1, None))


# problems on both sides of the automatic choice: one launch from the planes, the warp-level kernel, the expand pass
@pytest.mark.parametrize("M,N,K", [(64, 1024, 1024), (64, 1024, 8192), (512, 512, 4096), (1024, 1024, 512), (300, 2304, 1024), (2048, 2048, 256),
                                   (700, 1066, 2816), (96, 64, 16384)])
@pytest.mark.parametrize("wb,xb,sign", [(1, 1, "x"), (1, 2, "w"), (2, 1, "x"), (2, 2, "none")])
def test_automatic_choice(cuda_device, M, N, K, wb, xb, sign):
    import apnn_tc_b200 as ap
    rng = np.random.default_rng(M + 3 * N + K)
    W, _ = oracle.value_planes(rng, M, K, wb)
    X, _ = oracle.value_planes(rng, N, K, xb)
    v = oracle.gemm_popc(W, X, threads=8)
    if sign == "w":
        v = oracle.signed_correct(v, oracle.row_sums(X), 1)
    elif sign == "x":
        v = oracle.signed_correct(v, oracle.row_sums(W), 0)
    Wd, Xd = to_dev(W), to_dev(X)
    ws = torch.full((ap.gemm_workspace_bytes(M, N, K),), 0xEE, dtype=torch.uint8, device="cuda")
    got = ap.apmm(Wd, Xd, workspace=ws, epilogue=ap.make_epilogue("int32", signed=sign))
    ap.gemm_check(ws, M, N, K)
    assert np.array_equal(to_host(got, np.int32), v)
    if N % 32:
        return
    T = np.sort(rng.integers(int(v.min()) - 1, int(v.max()) + 2, size=(N, 3)), axis=1).astype(np.int32)
    for mode, bits in (("thresholds", 2), ("lowbits", 3)):
        got = ap.apmm(Wd, Xd, workspace=ws, epilogue=ap.make_epilogue(mode, bits, signed=sign, thresholds=to_dev(T)))
        ap.gemm_check(ws, M, N, K)
        assert np.array_equal(to_host(got), oracle.requant_pack(v, bits, 2 if mode == "thresholds" else 1, T))
