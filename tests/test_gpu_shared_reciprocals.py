"""The shared reciprocals of rp_math.cuh round as the plain operators do.

Roots and reciprocals are compared for every float. Quotients a / b are
compared for every divisor significand at the numerators whose quotient lies
nearest a rounding boundary (a 2^s = b M + d for an odd 25-bit M and small
d): the correction step is off by less than 3 / 2^49 of a unit there, so
only |d| <= 2 could round wrongly, and |d| <= 8 is run; subnormal quotients
next to the boundaries of their grid are run as well. Whole solves are
compared on random and degenerate matrices. Every comparison is of bits.
"""
import os
import subprocess

import pytest

from ropephysics_b200 import build

SOURCE = r"""
#include <cstdio>
#include <cuda_runtime.h>
#include "rp_internal.h"
#include "rp_math.cuh"
using namespace rp;
__device__ unsigned long long bad[4], used[4];
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__global__ void roots() {
    unsigned long long b0 = 0, b1 = 0, n0 = 0, n1 = 0;
    const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long u = blockIdx.x * blockDim.x + threadIdx.x; u < (1ull << 32); u += step) {
        const float a = __uint_as_float(unsigned(u));
        float s, y;
        bool ok = true;
        sqrtRecip(a, s, y, ok);
        if (ok) { ++n0; b0 += !(same(s, sqrtf(a)) && same(y, 1.0f / sqrtf(a))); }
        ok = true;
        const float r = recip(a, ok);
        if (ok) { ++n1; b1 += !same(r, 1.0f / a); }
    }
    atomicAdd(&bad[0], b0); atomicAdd(&used[0], n0);
    atomicAdd(&bad[1], b1); atomicAdd(&used[1], n1);
}
__global__ void quotients() {
    unsigned long long wrong = 0, n = 0;
    for (unsigned b = (1u << 23) + blockIdx.x * blockDim.x + threadIdx.x; b < (1u << 24); b += gridDim.x * blockDim.x) {
        const int t = __ffs(b) - 1;
        const unsigned odd = b >> t;
        unsigned inv = odd;
        for (int i = 0; i < 5; ++i) inv *= 2u - odd * inv;
        for (int s = 24; s <= 25; ++s)
            for (int d = -8; d <= 8; ++d) {
                if (d == 0 || (d & ((1 << t) - 1))) continue;
                const unsigned mod = 1u << (s - t);
                if (t >= s) continue;
                for (unsigned M = (unsigned(-(d >> t)) * inv) & (mod - 1u); M < (1u << 25); M += mod) {
                    if (M < (1u << 24) || !(M & 1u)) continue;
                    const unsigned long long num = (unsigned long long)b * M + (long long)d;
                    if (num & ((1ull << s) - 1ull)) continue;
                    const unsigned long long a = num >> s;
                    if (a < (1u << 23) || a >= (1u << 24)) continue;
                    // numerators from 2^-126 up to 2^63, divisors 2^-22 to 2^13
                    const float fa = float(unsigned(a)) * exp2f(float(int(b % 187u) - 149 + 2)) * (d & 1 ? -1.0f : 1.0f);
                    const float fb = float(b) * (M & 2u ? 0x1p-45f : 0x1p-10f);
                    bool ok = true;
                    const float q = quotient(fa, divisor(fb, recip(fb, ok)));
                    ++n;
                    wrong += !ok || !same(q, fa / fb);
                }
            }
        // subnormal quotients next to a boundary: a = b (2k + 1) 2^-150 cut to a
        // float, and its neighbour (b in [1, 2): no exact tie)
        const float fb = float(b) * 0x1p-23f;
        bool ok = true;
        const Divisor D = divisor(fb, recip(fb, ok));
        wrong += !same(quotient(0.0f, D), 0.0f) || !same(quotient(-0.0f, D), -0.0f);
        unsigned m = b * 2654435761u;
        for (int i = 0; i < 16; ++i) {
            m = m * 1664525u + 1013904223u;
            const unsigned a = unsigned(((unsigned long long)b * ((m >> (9 + i)) | 1u)) >> 24);
            for (unsigned e = 0; e < 2; ++e) {
                const float fa = __uint_as_float((a + e) | (m & 0x80000000u));
                wrong += !same(quotient(fa, D), fa / fb);
                ++n;
            }
        }
    }
    atomicAdd(&bad[2], wrong);
    atomicAdd(&used[2], n);
}
__device__ float draw(unsigned long long& x) {  // in (-1, 1)
    x = x * 6364136223846793005ull + 1442695040888963407ull;
    return float(int(x >> 32)) * 0x1p-31f;
}
__global__ void solves() {
    unsigned long long x = 977 + blockIdx.x * blockDim.x + threadIdx.x, wrong = 0, n = 0;
    for (int i = 0; i < 4096; ++i) {
        // J D J^T + alpha with scales over the projections' range, some
        // entries zero, some matrices singular or indefinite, some tiny
        M3 J;
        for (int r = 0; r < 3; ++r) for (int c = 0; c < 3; ++c) J.m[r][c] = (i & 7) == 1 && r != c ? 0.0f : draw(x);
        const float scale = exp2f(float((i >> 3) % 61 - 30));
        const V3 D{scale * fabsf(draw(x)), scale * fabsf(draw(x)), (i & 15) == 3 ? -scale : scale * fabsf(draw(x))};
        M3 A = sandwichDiag<false>(J, D);
        if ((i & 31) == 5) A = mscale(A, 0.0f);
        if ((i & 63) == 9) A.m[1][0] = A.m[0][1] = 1e-33f;
        if ((i & 63) == 12) { A.m[1][0] = draw(x) * 1e-37f; A.m[2][0] = draw(x) * 1e-25f; A.m[2][1] = draw(x) * 1e-37f; }
        if ((i & 63) == 10) A.m[2][0] = __int_as_float(0x7fc00000);
        V3 b{draw(x) * exp2f(float(i % 41 - 20)), (i & 3) ? draw(x) : 0.0f, draw(x)};
        if ((i & 63) == 11) b.y = __int_as_float(0x7f800000);
        if ((i & 63) == 12) b.x = b.y * 1e-30f;
        bool ok = true;
        const V3 y = solveSPD3Shared(A, b, ok);
        V3 z{0.0f, 0.0f, 0.0f};
        const bool solved = solveSPD3(A, b, z);
        if (ok) { ++n; wrong += !solved || !same(y.x, z.x) || !same(y.y, z.y) || !same(y.z, z.z); }
    }
    atomicAdd(&bad[3], wrong);
    atomicAdd(&used[3], n);
}
int main() {
    roots<<<1184, 256>>>();
    quotients<<<1184, 256>>>();
    solves<<<592, 256>>>();
    const cudaError_t e = cudaDeviceSynchronize();
    unsigned long long b[4], n[4];
    cudaMemcpyFromSymbol(b, bad, sizeof(b));
    cudaMemcpyFromSymbol(n, used, sizeof(n));
    for (int i = 0; i < 4; ++i) printf("%llu %llu\n", b[i], n[i]);
    return e == cudaSuccess ? 0 : 1;
}
"""

# how many inputs each comparison must have covered: the floats of
# [2^-100, 2^100], of [2^-62, 2^62], the near-boundary quotients, and most of
# the random solves
COVERED = [200 * (1 << 23), 124 * (1 << 23), 200_000_000, 592 * 256 * 4096 // 2]


@pytest.mark.gpu
def test_shared_reciprocals_round_as_the_operators(tmp_path):
    src, exe = tmp_path / "shared.cu", tmp_path / "shared"
    src.write_text(SOURCE)
    subprocess.run([build.NVCC, "-std=c++17", "-O3", "--fmad=false"] + build.ARCH +
                   ["-I" + os.path.join(build.CSRC), str(src), "-o", str(exe)], check=True, timeout=300)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    for (wrong, covered), need in zip(rows, COVERED):
        assert wrong == 0
        assert covered >= need, rows
