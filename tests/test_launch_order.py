"""Kernels launched as programmatic dependents may begin while the previous kernel of their stream still runs, and the
warp-level kernels let them begin before they have read anything.  So nothing global is read or written before the dependency
wait."""
import glob
import os
import re

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WAIT = re.compile(r"grid_dependency_wait\(\)|griddepcontrol\.wait")
# a store through a pointer parameter, a global store instruction, an atomic, or a TMA store
STORE = re.compile(r"\*p\.\w+ = |p\.\w+\[[^\]]*\] = |atomic\w+\(p\.|st\.global|cp\.async\.bulk\.tensor\.\dd\.global|__stcs|__stwt")
LOAD = re.compile(r"__ldg\(|ld\.global|tma_load_\dd\w*\(|load_2d<")


def kernels():
    for path in sorted(glob.glob(os.path.join(ROOT, "apnn_tc_b200", "csrc", "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__ void (?:__launch_bounds__\([^)]*(?:\([^)]*\)[^)]*)?\)\s*)?(\w+)\s*\(", text):
            start = text.index("{", text.index(")", m.end()))
            depth, i = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
                if depth == 0:
                    break
            yield os.path.basename(path), m.group(1), text[start:i]


def test_no_global_access_precedes_the_dependency_wait():
    seen = 0
    for path, name, body in kernels():
        wait = WAIT.search(body)
        if wait is None:      # not launched as a programmatic dependent
            continue
        seen += 1
        early = STORE.search(body[:wait.start()]) or LOAD.search(body[:wait.start()])
        assert early is None, f"{path}: {name} touches memory before its dependency wait: {body[early.start():early.start() + 60]!r}"
    assert seen >= 8


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(64, 128, 4096), (64, 1024, 1024)])
def test_status_flag_in_memory_the_previous_kernel_reads(cuda_device, M, N, K):
    """The status flag of an int8 GEMM in the block of the thresholds that the warp-level GEMM before it still reads: what a
    caching allocator does with a temporary that is freed between the two calls."""
    import apnn_tc_b200 as ap
    import oracle
    from gpu_util import to_dev, to_host
    rng = np.random.default_rng(M + N)
    W, wl = oracle.value_planes(rng, M, K, 1)
    X, xl = oracle.value_planes(rng, N, K, 2)
    v = oracle.gemm_popc(W, X, threads=8)
    T = np.sort(rng.integers(int(v.min()), int(v.max()) + 1, size=(N, 3)), axis=1).astype(np.int32)
    T[0] = int(v[:, 0].max()) + 1          # no value of column 0 reaches a threshold, every one reaches 0
    want = oracle.requant_pack(v, 2, 2, T)
    Wd, Xd, T0, Td = to_dev(W), to_dev(X), to_dev(T), to_dev(T)
    A8, B8 = torch.ones((128, 128), dtype=torch.uint8, device="cuda"), torch.ones((64, 128), dtype=torch.uint8, device="cuda")
    D8 = torch.empty((128, 64), dtype=torch.int32, device="cuda")
    outs = [torch.zeros((2, M, N // 32), dtype=torch.int32, device="cuda") for _ in range(20)]
    for out in outs:
        Td.copy_(T0)
        ap.apmm(Wd, Xd, out, algo="imma", epilogue=ap.make_epilogue("thresholds", 2, thresholds=Td))
        ap.gemm_i8(A8, B8, D8, status_flag=Td.view(-1)[:1])
    for out in outs:
        assert np.array_equal(to_host(out), want)
    assert int(Td.view(-1)[0].item()) == 0 and bool((D8 == 128).all())
