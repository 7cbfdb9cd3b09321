"""The FP64 <-> FP32 conversions on the integer pipe (device_common.cuh) against
the casts, bit for bit (GPU): every exponent and sign with mantissas at ties of
both parities, their neighbours, carries into the exponent and all ones, and
random values."""
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include "device_common.cuh"

// mantissas: FP32 part x the 29 bits below it
__constant__ unsigned high[8] = {0u, 1u, 2u, 3u, 0x2aaaaau, 0x400000u, 0x7ffffeu, 0x7fffffu};
__constant__ unsigned low[8] = {0u, 1u, 0x0fffffffu, 0x10000000u, 0x10000001u, 0x1ffffffeu, 0x1fffffffu, 0x12345678u};
constexpr unsigned LISTED = 2048u * 2u * 64u, RANDOM = 1u << 22;

__global__ void compare(unsigned *wrong)
{
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= LISTED + RANDOM) return;
    unsigned long long u;
    if (t < LISTED) {
        const unsigned long long m = ((unsigned long long)high[t & 7u] << 29) | low[t >> 3 & 7u];
        u = ((unsigned long long)(t >> 6) << 52) | m;  // 11 bits of exponent, the sign above them
    } else {  // splitmix64
        u = (t - LISTED + 1ull) * 0x9e3779b97f4a7c15ull;
        u = (u ^ (u >> 30)) * 0xbf58476d1ce4e5b9ull;
        u = (u ^ (u >> 27)) * 0x94d049bb133111ebull;
        u ^= u >> 31;
    }
    const double v = __longlong_as_double((long long)u);
    const float f = (float)v;
    if (__float_as_uint(lss::to_float(v)) != __float_as_uint(f)) atomicAdd(wrong, 1u);
    if (__double_as_longlong(lss::to_double(f)) != __double_as_longlong((double)f)) atomicAdd(wrong + 1, 1u);
    const float2 s = lss::split_double(v);
    const float l = (float)(v - (double)f);
    if (__float_as_uint(s.x) != __float_as_uint(f) || __float_as_uint(s.y) != __float_as_uint(l)) atomicAdd(wrong + 2, 1u);
}

int main()
{
    unsigned *d = nullptr, h[3] = {~0u, ~0u, ~0u};
    if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return 1;
    compare<<<(LISTED + RANDOM + 255) / 256, 256>>>(d);
    if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    std::printf("%u %u %u\n", h[0], h[1], h[2]);
    return 0;
}
"""


def test_conversions_equal_the_casts(built, tmp_path):
    from lss import _paths, build
    src, exe = tmp_path / "compare.cu", tmp_path / "compare"
    src.write_text(SOURCE)
    subprocess.run([build._nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-I", _paths.CSRC, "-I", _paths.INCLUDE,
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0", "0", "0"], out
