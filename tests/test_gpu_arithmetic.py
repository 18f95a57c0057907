"""The device helpers that stand in for division, against the division operator and roundf on the same GPU, bit for bit.  The
helpers are compiled from the library's own header."""
import ctypes as C
import os
import shutil
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu
HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chimere_b200", "csrc", "common.cuh")
SOURCE = r"""
#include "HEADER"
using namespace chimere;
__device__ bool same(float a, float b) { return (a != a && b != b) || __float_as_uint(a) == __float_as_uint(b); }
// every float g: the bits of silu_mul_ref from -87 on and below -88.8; between, where the quotient leaves the normal numbers, as small as it
__global__ void silu_kernel(unsigned long long* bad) {
    for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < (1ull << 32); i += gridDim.x * 256ull) {
        const float g = __uint_as_float((unsigned)i), w = silu_mul_ref(g, 1.0f), v = silu_mul_fast(g, 1.0f);
        const bool tail = g < -87.0f && g > -88.8f, zero = v == 0.0f && w == 0.0f;
        if (!same(w, v) && !zero && !(tail && v <= 0.0f && v >= -2.5e-36f)) atomicAdd(bad, 1ull);
    }
}
extern "C" int silu_check(unsigned long long* bad) { silu_kernel<<<1184, 256>>>(bad); return (int)cudaDeviceSynchronize(); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = os.environ.get("NVCC", "nvcc")
    if shutil.which(nvcc) is None:
        pytest.skip("nvcc is not installed")
    d = tmp_path_factory.mktemp("arithmetic")
    (d / "check.cu").write_text(SOURCE.replace("HEADER", HEADER))
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--compiler-options", "-fPIC", "-shared", "-o",
                    str(d / "check.so"), str(d / "check.cu")], check=True)
    return C.CDLL(str(d / "check.so"))


def _mismatches(check):
    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    assert check(C.c_void_p(bad.data_ptr())) == 0
    return int(bad.item())


def test_silu_is_the_reference_quotient_for_every_float(lib):
    assert _mismatches(lib.silu_check) == 0
