"""GELU's reciprocal (an approximation and one Newton step) against CUDA's correctly rounded one, bit for bit."""
import ctypes
import os
import shutil
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "orion_b200", "csrc", "kernels")

SOURCE = r"""
#include "fast_gelu.cuh"
__global__ void compare(unsigned first, unsigned long long count, unsigned long long* differ) {
    unsigned long long mine = 0;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < count; i += (unsigned long long)gridDim.x * blockDim.x) {
        const float x = __uint_as_float(first + (unsigned)i);
        mine += __float_as_uint(ob200::reciprocal_from_1(x)) != __float_as_uint(__frcp_rn(x));
    }
    if (mine) atomicAdd(differ, mine);
}
__global__ void evaluate(const float* x, float* y, int n) {
    if (threadIdx.x < n) y[threadIdx.x] = ob200::reciprocal_from_1(x[threadIdx.x]);
}
extern "C" int run_compare(unsigned first, unsigned long long count, unsigned long long* differ) {
    compare<<<592, 256>>>(first, count, differ);
    return (int)cudaDeviceSynchronize();
}
extern "C" int run_evaluate(const float* x, float* y, int n) {
    evaluate<<<1, 32>>>(x, y, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("reciprocal")
    (d / "reciprocal.cu").write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "--cudart", "shared", "-shared",
                    "-I", KERNELS, "-o", str(d / "reciprocal.so"), str(d / "reciprocal.cu")], check=True)
    torch.cuda.init()
    L = ctypes.CDLL(str(d / "reciprocal.so"))
    L.run_compare.argtypes = [ctypes.c_uint, ctypes.c_ulonglong, ctypes.c_void_p]
    L.run_evaluate.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]
    return L


def test_every_float_from_1_to_64_gives_the_correctly_rounded_reciprocal(lib):
    """64 is 1 + 0.3275911 |a| / sqrt 2 for |a| = 272, where exp(-a^2 / 2) has long been zero."""
    differ = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    first, last = 0x3f800000, 0x42800000
    assert lib.run_compare(first, last - first + 1, differ.data_ptr()) == 0
    assert differ.item() == 0


def test_beyond_64(lib):
    """Large arguments, infinity and NaN: the approximation's own zero where the reciprocal is subnormal, no NaN but from NaN."""
    x = torch.tensor([64.5, 1e6, 9.9e29, 1e30, 8e37, 3e38, float("inf"), float("nan")], device="cuda")
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    assert lib.run_evaluate(x.data_ptr(), y.data_ptr(), x.numel()) == 0
    got = y.cpu().tolist()
    for a, b in zip(x.cpu().tolist()[:5], got):
        assert abs(a * b - 1.0) < 3e-7   # one ulp of the approximation and the rounding of the product
    assert 0.0 <= got[5] < 4e-39 and got[6] == 0.0 and got[7] != got[7]
