"""recip2 and div2 (paired FP32 reciprocals and quotients of the IEEE kernels)
against __frcp_rn and __fdiv_rn, bit for bit: reciprocals of every significand in
every exponent of their range, quotients of hashed operands over theirs, its ends
and the significands next to a power of two among them, both signs.  Compiled from
the kernels' own header, as the library compiles it."""
import importlib.util
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

CU = r'''
#include <cstdio>
#define GBT_ARITH_NS checked
#include "gbt_kernels.cuh"
using namespace gbt::checked;

__device__ unsigned long long g_bad[2];

__device__ __forceinline__ float number(uint32_t sign, int exponent, uint32_t significand) {
    return __uint_as_float(sign << 31 | (uint32_t)(exponent + 127) << 23 | (significand & 0x7fffffu));
}
__device__ __forceinline__ uint32_t mix(unsigned long long x) {   // splitmix64
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ x >> 30) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ x >> 27) * 0x94d049bb133111ebull;
    return (uint32_t)((x ^ x >> 31) >> 16);
}

// every significand at exponents -14 .. 29, and at 30 the power of two
__global__ void reciprocals() {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;   // 2^23
    unsigned bad = 0;
    for (int e = -14; e <= 30; ++e)
        for (uint32_t sign = 0; sign < 2; ++sign) {
            const float b0 = number(sign, e, e == 30 ? 0u : s), b1 = number(sign ^ 1u, -e / 2, s ^ 0x2aaaaau);
            const f2 r = recip2(f2_pack(b0, b1), f2_pack(-b0, -b1));
            bad += __float_as_uint(f2_lo(r)) != __float_as_uint(__frcp_rn(b0));
            bad += __float_as_uint(f2_hi(r)) != __float_as_uint(__frcp_rn(b1));
        }
    if (bad) atomicAdd(&g_bad[0], bad);
}

__device__ __forceinline__ uint32_t edge_or(uint32_t choice, uint32_t significand) {
    switch (choice & 15u) {   // one in four next to a power of two
        case 0: return 0u;
        case 1: return 1u;
        case 2: return 0x7fffffu;
        case 3: return 0x7ffffeu;
        default: return significand;
    }
}

__global__ void quotients(unsigned long long seed) {
    const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned bad = 0;
    float a[2], b[2];
    for (int k = 0; k < 64; ++k) {
        for (int j = 0; j < 2; ++j) {
            const unsigned long long n = seed + ((i * 64 + k) * 2 + j) * 4;
            const uint32_t h = mix(n), g = mix(n + 1);
            int ea = (int)(mix(n + 2) % 161u) - 80, eb = (int)(mix(n + 3) % 45u) - 14;
            if ((h >> 28) == 0u) ea = h >> 27 & 1u ? 80 : -80;
            if ((g >> 28) == 0u) eb = g >> 27 & 1u ? 30 : -14;
            a[j] = number(h >> 26 & 1u, ea, ea == 80 ? 0u : edge_or(h >> 22, h));
            b[j] = number(g >> 26 & 1u, eb, eb == 30 ? 0u : edge_or(g >> 22, g));
        }
        const f2 B = f2_pack(b[0], b[1]), nb = f2_pack(-b[0], -b[1]);
        const f2 q = div2(f2_pack(a[0], a[1]), nb, recip2(B, nb));
        bad += __float_as_uint(f2_lo(q)) != __float_as_uint(__fdiv_rn(a[0], b[0]));
        bad += __float_as_uint(f2_hi(q)) != __float_as_uint(__fdiv_rn(a[1], b[1]));
    }
    if (bad) atomicAdd(&g_bad[1], bad);
}

int main() {
    reciprocals<<<(1 << 23) / 256, 256>>>();
    for (int k = 0; k < 8; ++k) quotients<<<1 << 15, 256>>>(0x5eedull + ((unsigned long long)k << 40));   // 8.6 G
    unsigned long long bad[2] = {1, 1};
    const cudaError_t e = cudaMemcpyFromSymbol(bad, g_bad, sizeof(bad));
    std::printf("%s %llu %llu\n", cudaGetErrorString(e), bad[0], bad[1]);
    return e != cudaSuccess;
}
'''


def test_paired_reciprocals_and_quotients(gpu, tmp_path):
    path = os.path.join(HERE, "..", "cu-reconstruction_gb300", "build.py")
    spec = importlib.util.spec_from_file_location("gbt_engine_build", path)
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    src, exe = str(tmp_path / "divides.cu"), str(tmp_path / "divides")
    with open(src, "w") as f:
        f.write(CU)
    subprocess.check_call([build.nvcc()] + build.ARCH + build.COMMON + build.UNITS["k_ieee.cu"] +
                          ["-I" + build.CSRC, src, "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "no error 0 0", r.stdout + r.stderr
