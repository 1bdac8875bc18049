"""The branch-free quotients and roots of gbl_math.cuh against CUDA's own.

recipNearest over every mantissa, rootNearest over every mantissa of an even
and an odd exponent, each at several exponents of their range; quotient() over
the pairs whose exact quotient lies within 32 / (2 b) of an ulp from a midpoint
(in integers, |2 a 2^k - b (2 m + 1)| <= 32: the only ones an error below
2^-22 ulp before the last rounding could round wrongly), enumerated divisor by
divisor, and over random pairs across the accepted ranges and the signed zeros.
Equality is exact.
"""
import subprocess

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include "gbl_math.cuh"
#include <cstdio>
using namespace gbl;
using ull = unsigned long long;
__device__ void note(ull *bad, int k, float got, float want) {
    if (__float_as_uint(got) != __float_as_uint(want)) atomicAdd(bad + k, 1ULL);
}
__global__ void reciprocals(ull *bad, int exponent) {
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    const float b = __uint_as_float((unsigned(127 + exponent) << 23) | m);
    if (!divisorOk(b)) atomicAdd(bad + 0, 1ULL);
    note(bad, 0, recipNearest(b), __frcp_rn(b));
}
__global__ void roots(ull *bad, int exponent) {
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    const float s = __uint_as_float((unsigned(127 + exponent) << 23) | m);
    if (!rootOk(s)) atomicAdd(bad + 1, 1ULL);
    note(bad, 1, rootNearest(s), __fsqrt_rn(s));
}
// QuickMath::root scales what is below 2^-60: zero, every denormal exponent's
// mantissas and the normals up to there.
__global__ void tinyRoots(ull *bad, unsigned first) {
    const float s = __uint_as_float(first + blockIdx.x * blockDim.x + threadIdx.x);
    QuickMath m;
    note(bad, 1, m.root(s), __fsqrt_rn(s));
    if (!m.good) atomicAdd(bad + 1, 1ULL);
}
__global__ void midpoints(ull *bad, ull *tried) {
    const unsigned B = (1U << 23) | (blockIdx.x * blockDim.x + threadIdx.x);
    const float b = __uint_as_float(0x3f800000U | (B & 0x7fffffU)), y = recipNearest(b);
    const int t = __ffs(B) - 1;
    if (t > 5) return;
    const unsigned Bp = B >> t;
    for (int shift = 23; shift <= 24; ++shift)
        for (int r = -(32 >> t); r <= (32 >> t); ++r) {
            if (!(r & 1)) continue;
            const long long half = (static_cast<long long>(r) + Bp) / 2;
            long long x = ((half % Bp) + Bp) % Bp;
            for (int k = 0; k < shift - t; ++k) x = (x & 1) ? (x + Bp) / 2 : x / 2;
            for (ull A = x; A < (1ULL << 24); A += Bp) {
                if (A < (1ULL << 23) || (shift == 23 ? A < B : A >= B)) continue;
                const float a = __uint_as_float(0x3f800000U | (unsigned(A) & 0x7fffffU));
                atomicAdd(tried, 1ULL);
                note(bad, 2, quotient(a, b, y), __fdiv_rn(a, b));
            }
        }
}
__device__ ull mix(ull z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}
__global__ void pairs(ull *bad, int n) {
    const ull t = blockIdx.x * static_cast<ull>(blockDim.x) + threadIdx.x;
    for (int i = 0; i < n; ++i) {
        const ull z = mix(t * 0x9E3779B97F4A7C15ULL + i), w = mix(z + 1);
        const float b = __uint_as_float((unsigned(127 - 90 + w % 120) << 23) | unsigned(z & 0x7fffff));
        float a = __uint_as_float((unsigned(127 - 90 + (w >> 16) % 120) << 23) | unsigned((z >> 23) & 0x7fffff));
        if ((w >> 40) % 64 == 0) a = 0.0F;
        if ((w >> 50) & 1) a = -a;
        if (!divisorOk(b) || dividendKey(a) < kDividendLeast) atomicAdd(bad + 3, 1ULL);
        const float want = __fdiv_rn(a, b);
        if (a != 0.0F && !(fabsf(want) >= 0x1p-120F && fabsf(want) < 0x1p100F)) continue;
        note(bad, 3, quotient(a, b, recipNearest(b)), want);
    }
}
int main() {
    ull *c;
    cudaMallocManaged(&c, 8 * sizeof(ull));
    for (int k = 0; k < 8; ++k) c[k] = 0;
    const int divisors[] = {-90, -40, -1, 0, 1, 29}, radicands[] = {-100, -99, -78, -77, -20, -19, 0, 1, 58, 59};
    for (int e : divisors) reciprocals<<<(1 << 23) / 256, 256>>>(c, e);
    for (int e : radicands) roots<<<(1 << 23) / 256, 256>>>(c, e);
    for (unsigned e : {0U, 1U, 2U, 30U, 66U, 67U, 68U}) tinyRoots<<<(1 << 23) / 256, 256>>>(c, e << 23);
    midpoints<<<(1 << 23) / 256, 256>>>(c, c + 4);
    pairs<<<1024, 256>>>(c, 2000);
    const cudaError_t e = cudaDeviceSynchronize();
    std::printf("%d %llu %llu %llu %llu %llu\n", static_cast<int>(e), c[0], c[1], c[2], c[3], c[4]);
    return 0;
}
"""


def test_quotients_and_roots_are_correctly_rounded(device, tmp_path):
    from banjo_gb300 import build

    src, exe = tmp_path / "division.cu", tmp_path / "division"
    src.write_text(PROGRAM)
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", *build.DEVICE_FP, "-I", build.CSRC, str(src), "-o",
                    str(exe)], check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout.split()
    error, recips, roots, midpoints, pairs, tried = (int(x) for x in out)
    assert error == 0
    assert tried > 180_000_000
    assert (recips, roots, midpoints, pairs) == (0, 0, 0, 0)
