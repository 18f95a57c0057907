"""Device helpers of the library's own header, compiled into kernels of their own: those that stand in for division against the division
operator and roundf on the same GPU, bit for bit, and the bounded wait."""
import ctypes as C
import os
import shutil
import subprocess
import time

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
// one block of 32 values per warp: Q8_1 with the division operator, fmaxf over the block (NaN left out) and roundf
__device__ unsigned mix(unsigned long long x) {
    x ^= x >> 33; x *= 0xff51afd7ed558ccdull; x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ull; x ^= x >> 33;
    return (unsigned)x;
}
__global__ void q8_kernel(unsigned long long* bad) {
    const int lane = threadIdx.x & 31;
    for (unsigned long long blk = blockIdx.x * 8ull + (threadIdx.x >> 5); blk < (1ull << 24); blk += gridDim.x * 8ull) {
        const unsigned hb = mix(2 * blk + 1), h = mix((blk * 32 + lane) * 2);
        // the block's magnitude: all of the floats', with the limits of the fast form among them; its values: uniform, around the
        // half-way points, far smaller, zeros, infinities, NaN
        float top = __uint_as_float((hb >> 1) & 0x7FFFFFFFu);
        if ((hb & 7) == 1) top = 1e-25f * (1.0f + (float)(hb >> 20) * 1e-6f);
        if ((hb & 7) == 2) top = 1e25f * (1.0f - (float)(hb >> 20) * 1e-6f);
        if ((hb & 7) > 3) top = (float)(hb >> 8) * 1e-5f;
        const float step = top / 127.0f;
        float v = top * ((float)(h >> 8) / 16777216.0f);
        if ((hb & 24) == 8) v = step * ((float)(h % 127) + 0.5f) * (1.0f + (float)((int)(h >> 16) % 5 - 2) * 5.9e-8f);
        if ((hb & 24) == 16 && lane > 3) v *= 1e-30f;
        if ((hb & 96) == 32 && (h & 31) == 0) v = __uint_as_float(0x7FC00000u);
        if ((hb & 480) == 64 && lane == (hb >> 27)) v = __uint_as_float(0x7F800000u);
        if ((hb & 0xF00) == 0 && (h & 3)) v = 0.0f;
        if ((hb & 0xFFF000) == 0) v = (hb >> 24) & 1 ? 0.0f : __uint_as_float(0x7FC00000u);
        if (lane == 5 && !((hb >> 11) & 1)) v = top;
        if (h & 0x800000u) v = -v;
        float d;
        const int8_t q = q8_1_warp(v, d);
        float amax = fabsf(v);
        for (int m = 16; m > 0; m >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
        const float dp = amax / 127.0f;
        const int8_t qp = amax == 0.0f ? (int8_t)0 : (int8_t)roundf(v / dp);
        if (q != qp || !same(d, dp)) atomicAdd(bad, 1ull);
    }
}
extern "C" int q8_check(unsigned long long* bad) { q8_kernel<<<1184, 256>>>(bad); return (int)cudaDeviceSynchronize(); }
// a wait on a barrier that nobody arrives at: comes back with false
__global__ void wait_kernel(unsigned long long* bad) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) { mbar_init(&bar, 1); mbar_fence_init(); }
    __syncthreads();
    if (mbar_wait(&bar, 0)) atomicAdd(bad, 1ull);
}
extern "C" int wait_check(unsigned long long* bad) { wait_kernel<<<1, 32>>>(bad); return (int)cudaDeviceSynchronize(); }
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


def test_q8_1_blocks_are_those_of_the_plain_operations(lib):
    assert _mismatches(lib.q8_check) == 0


@pytest.mark.parametrize("T", [3, 40, 200])
def test_routers_and_operator_quantise_alike(T):
    """The Q8_1 rows that the routers leave and those of the operator entry are the same bytes, NaN, infinities and extremes included."""
    from chimere_b200 import abi, configs
    from chimere_b200.layer import MoeScratch, MoeWeightsTiled, route_only
    cfg = configs.scaled(configs.QWEN_Q4_0, E=256, H=512, F=64, F_s=0)
    tiled = MoeWeightsTiled(configs.make_layer(cfg, device="cuda"))
    x = configs.make_input(cfg, T, device="cuda")
    x[0, 3], x[0, 40], x[0, 41], x[1, 70] = float("nan"), float("inf"), float("-inf"), 1e30
    x[1, 96:128], x[1, 128:160], x[2, :32] = float("nan"), 0.0, torch.arange(32, device="cuda") * 1e-28
    x[2, 64:96] = torch.arange(32, device="cuda") + 0.5
    x[2, 64] = 127.0
    sc = MoeScratch(tiled, T)
    route_only(tiled, sc, x)
    want = torch.zeros(T, 512 // 32 * 36, dtype=torch.uint8, device="cuda")
    abi.load().chimere_quantize_q8_1_batched(x.data_ptr(), want.data_ptr(), 512, 512, T, torch.cuda.current_stream().cuda_stream)
    assert torch.equal(sc.x_q8(T), want)


def test_a_wait_that_nobody_ends_gives_up_within_seconds(lib):
    torch.cuda.synchronize()
    start = time.monotonic()
    assert _mismatches(lib.wait_check) == 0
    assert time.monotonic() - start < 5.0
