"""Every function declared in include/*.h is exported by its library (no compute calls)."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADERS = {"orion_sched.h": "liborion_sched.so", "orion_capture.h": "liborion_capture.so", "orion_kernels.h": "liborion_kernels.so"}


def _declared(header):
    text = open(os.path.join(ROOT, "include", header)).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    names = re.findall(r"\b([A-Za-z_][A-Za-z0-9_]*)\s*\([^;{]*\)\s*;", text)
    return sorted(set(n for n in names if n not in ("defined",)))


@pytest.mark.parametrize("header", sorted(HEADERS))
def test_library_exports_every_declared_symbol(header, built):
    names = _declared(header)
    assert len(names) >= 5
    lib = ctypes.CDLL(built[HEADERS[header]])
    missing = [n for n in names if not hasattr(lib, n)]
    assert not missing, "not exported by %s: %s" % (HEADERS[header], missing)


def test_reference_entry_points_are_present(built):
    sched = ctypes.CDLL(built["liborion_sched.so"])
    for name in ("sched_init", "setup", "setup_change", "schedule", "reset"):
        assert hasattr(sched, name)
    cap = ctypes.CDLL(built["liborion_capture.so"])
    for name in ("block", "stop", "cudaLaunchKernel", "cudaMemcpyAsync", "cudaMalloc", "cublasSgemm_v2",
                 "cublasSgemmStridedBatched", "cudnnConvolutionForward", "cudnnBatchNormalizationForwardInference",
                 "cudnnBackendExecute", "cublasGemmEx", "cublasLtMatmul", "cudaLaunchKernelExC", "cudaMallocAsync", "cudaFreeAsync",
                 "cudaMallocManaged", "cudaGraphLaunch"):
        assert hasattr(cap, name), name


def test_kernel_entry_points_reject_bad_arguments_without_a_gpu(built):
    lib = ctypes.CDLL(built["liborion_kernels.so"])
    # dtype 7 does not exist; argument checks run before any CUDA call
    rc = lib.ob200_conv2d_fprop_ex(None, None, None, None, None, None, 0, 7, 1, 8, 8, 8, 8, 1, 1, 1, 1, 0, 0, 1, 1, 128, 1, None,
                                   None, 8, None)
    assert rc < 0
    bn, splits = ctypes.c_int(), ctypes.c_int()
    lib.ob200_plan_conv.argtypes = [ctypes.c_int, ctypes.c_longlong] + [ctypes.c_int] * 5 + [ctypes.POINTER(ctypes.c_int)] * 2
    assert lib.ob200_plan_conv(0, 196, 512, 3, 3, 512, 148, ctypes.byref(bn), ctypes.byref(splits)) == 0
    assert bn.value in (64, 128) and 1 <= splits.value <= 16


def _plan(lib, dtype, M, Kout, R, S, C, ctas):
    bn, splits, sk = ctypes.c_int(), ctypes.c_int(), ctypes.c_int()
    lib.ob200_plan_schedule.argtypes = [ctypes.c_int, ctypes.c_longlong] + [ctypes.c_int] * 5 + [ctypes.POINTER(ctypes.c_int)] * 3
    assert lib.ob200_plan_schedule(dtype, M, Kout, R, S, C, ctas, ctypes.byref(bn), ctypes.byref(splits), ctypes.byref(sk)) == 0
    return bn.value, splits.value, sk.value


def test_schedule_planning_host_logic(built):
    """Which schedule a problem gets is host arithmetic: checked here for the ResNet-50 shapes without a GPU."""
    lib = ctypes.CDLL(built["liborion_kernels.so"])
    # deep tiles with a ragged last wave at training batch size: stream-K (196 tiles of 36 k-blocks on 148 CTAs)
    assert _plan(lib, 0, 32 * 28 * 28, 128, 3, 3, 128, 148) == (128, 1, 1)
    # shallow 1x1 layer (2 k-blocks per tile): one unit per tile, wide tiles, never cut
    assert _plan(lib, 0, 32 * 56 * 56, 256, 1, 1, 64, 148) == (128, 1, 0)
    # batch-4 inference, few deep tiles: split-K over the idle SMs, chains of at least four k-blocks
    bn, splits, sk = _plan(lib, 0, 4 * 7 * 7, 512, 3, 3, 512, 148)
    assert sk == 0 and bn == 64 and 2 <= splits <= 16 and 144 // splits >= 4
    # narrow outputs take narrow tiles; a small SM quota never over-splits
    assert _plan(lib, 0, 32 * 56 * 56, 64, 1, 1, 256, 148)[0] == 64
    for ctas in (1, 8, 37, 148):
        for (M, Kout, R, C) in [(12544, 64, 3, 64), (784, 1024, 1, 256), (196, 2048, 1, 512), (100352, 64, 7, 4)]:
            bn, splits, sk = _plan(lib, 0, M, Kout, R, R, C, ctas)
            nk = R * ((R * C + 31) // 32)
            assert bn in (64, 128) and 1 <= splits <= max(1, nk) and sk in (0, 1)
            tiles = ((M + 127) // 128) * ((Kout + bn - 1) // bn)
            if sk:
                assert splits == 1 and tiles * 4 >= ctas and nk >= 8
            else:
                assert tiles * splits <= max(tiles, ctas)
    # bad arguments are rejected
    assert lib.ob200_plan_schedule(0, 0, 64, 1, 1, 64, 148, None, None, None) < 0


def _gemm_plan(lib, M, N, K, batch=1, tri=0, ctas=148):
    out = [ctypes.c_int() for _ in range(4)]
    lib.ob200_plan_gemm_bf16.argtypes = [ctypes.c_int] * 3 + [ctypes.c_longlong] + [ctypes.c_int] * 2 + [ctypes.POINTER(ctypes.c_int)] * 4
    assert lib.ob200_plan_gemm_bf16(M, N, K, batch, tri, ctas, *[ctypes.byref(o) for o in out]) == 0
    return [o.value for o in out]


@pytest.mark.parametrize("M,N,K,batch,tri", [(1, 8, 8, 1, 0), (77, 768, 768, 1, 0), (129, 64, 4096, 1, 0), (600, 1024, 4096, 1, 0), (3072, 2304, 768, 1, 0),
                                             (8192, 32000, 1024, 1, 0), (1024, 1024, 64, 32, 1), (512, 64, 512, 256, 2), (768, 768, 8192, 1, 0)])
def test_gemm_plan_keeps_to_the_quota_and_to_one_split(built, M, N, K, batch, tri):
    """At most `num_ctas` CTAs, pairs whole, and a split factor (the order of the sums) that no quota changes."""
    lib = ctypes.CDLL(built["liborion_kernels.so"])
    splits = _gemm_plan(lib, M, N, K, batch, tri)[2]
    for ctas in list(range(1, 18)) + [33, 79, 80, 147, 148, 200]:
        bn, cg, sp, grid = _gemm_plan(lib, M, N, K, batch, tri, ctas)
        assert sp == splits and 1 <= grid <= ctas and grid % cg == 0
        assert bn in ((64,) if N <= 64 else (128, 256)) and not (cg == 2 and (M <= 128 or tri)) and not (bn == 256 and N < 256)
    assert _gemm_plan(lib, M, N, K, batch, tri, 1)[1] == 1


@pytest.mark.parametrize("M,N,K", [(2048, 768, 3072), (3072, 768, 8192), (768, 3072, 8192), (2304, 768, 8192), (1232, 1024, 4096)])
def test_gemm_plan_does_not_cut_a_reduction_whose_tiles_fill_the_device(built, M, N, K):
    """Tiles of 128 x 128 occupy more than half of 148 SMs: a second launch and partial matrices cost more than they give."""
    lib = ctypes.CDLL(built["liborion_kernels.so"])
    assert _gemm_plan(lib, M, N, K)[2] == 1


def test_gemm_plan_gives_shallow_products_single_ctas(built):
    """A 64-deep product is bound by its tiles' way out of tensor memory, which pairs do not shorten."""
    lib = ctypes.CDLL(built["liborion_kernels.so"])
    assert _gemm_plan(lib, 512, 512, 64, 256)[:2] == [256, 1]
    assert _gemm_plan(lib, 3072, 1024, 72)[1] == 1
    assert _gemm_plan(lib, 8192, 4096, 1024)[:2] == [256, 2]   # a deep one is not
    assert _gemm_plan(lib, 3072, 2304, 768, ctas=3)[1] == 1    # two of three CTAs would work


def test_filter_gradient_ranges(built):
    """Long reductions of few tiles take two rounds of the device, shorter ones one; none is cut into ranges of one k-block."""
    lib = ctypes.CDLL(built["liborion_kernels.so"])
    plan = lib.ob200_plan_wgrad_splits
    plan.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    assert plan(1, 25088, 148) == 296
    assert plan(2, 221, 148) == 74 and plan(1, 392, 148) == 148 and plan(2, 10, 148) == 5 and plan(36, 20, 148) == 9 and plan(4, 220, 148) == 74
    for tiles in (1, 2, 3, 9, 300):
        for kblocks in (1, 2, 7, 130, 255, 257, 1000, 30000):
            for ctas in (1, 7, 148):
                n = plan(tiles, kblocks, ctas)
                assert 1 <= n <= max(1, kblocks // 2) and (n - 1) * tiles < 2 * ctas
                assert 4 * n <= kblocks or n * tiles <= ctas or ctas // tiles <= 64
