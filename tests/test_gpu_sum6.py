"""The six-value neighbour sum on the integer and FP32 pipes (sum6_int,
nyx_gb300/csrc/pm_sum6.cuh) against the FP64 additions it replaces, bit for bit
(tolerance: exact).

A probe compiled here draws sets of doubles from a hash of the index: values of
one or of mixed signs, 0 to 6 and 7 and more binades apart (the edge of the integer
path and beyond it), fractions of all zeros, all ones, a few low bits, a few high
bits (ties and carries), exact negatives of the value before (cancellation to zero),
zeros of both signs, and every exponent (subnormals, overflow, infinities, NaNs: a
NaN equals a NaN of any payload).
"""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <cstdio>
#include "pm_sum6.cuh"
using namespace nyxpm;
typedef unsigned long long u64;

__device__ __forceinline__ u64 mix64(u64 z)
{
    z += 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

constexpr int kKinds = 10;

__device__ bool differ(double x, double y)
{
    return !(x != x && y != y) && __double_as_longlong(x) != __double_as_longlong(y);
}

__global__ void check(int kind, u64 total, u64* bad)
{
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < total; i += (u64)gridDim.x * blockDim.x) {
        const u64 h = mix64(i * 16 + kind);
        const int signs = (int)(h >> 16) & 3;      // 0: all plus, 1: all minus, else mixed
        u64 e0 = 1000;
        if (kind == 8) e0 = (h >> 32) % 2047;       // every exponent
        if (kind == 9) e0 = 55 + (h >> 32) % 20;    // the lower edge of the integer path
        double v[6];
        for (int c = 0; c < 6; ++c) {
            const u64 r = mix64(h + c * 0x1234567ULL);
            u64 e = e0;
            if (kind == 1) e += r % 2;
            if (kind == 2 || kind == 9) e += r % 7;
            if (kind == 3) e += 6 * (r & 1);
            if (kind == 4) e += 7 * (r & 1);
            if (kind == 5) e += r % 70;
            if (kind == 8) e += r % 9;
            if (e > 2047) e = 2047;
            u64 m = (r >> 8) & 0xfffffffffffffULL;
            switch ((r >> 61) & 7) {
            case 0: m = 0; break;
            case 1: m = 0xfffffffffffffULL; break;
            case 2: m &= ~0xffULL; break;
            case 3: m &= 3; break;
            case 4: m |= 0xfffffffffff00ULL; break;
            }
            const u64 sg = signs < 2 ? (u64)signs : (r >> 60) & 1;
            u64 bits = (sg << 63) | (e << 52) | m;
            if (kind == 6 && (r & 0x30) == 0) bits = sg << 63;
            if (kind == 7 && c && (r & 0x30)) bits = (u64)__double_as_longlong(-v[c - 1]);
            v[c] = __longlong_as_double((long long)bits);
        }
        if (differ(sum6_int(v), sum6(v, false))) atomicAdd(bad + kind, 1ULL);
    }
}

int main()
{
    u64* bad;
    cudaMalloc(&bad, kKinds * sizeof(u64));
    cudaMemset(bad, 0, kKinds * sizeof(u64));
    for (int kind = 0; kind < kKinds; ++kind) check<<<1024, 256>>>(kind, 1ULL << 24, bad);
    u64 h[kKinds];
    if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    int rc = 0;
    for (int kind = 0; kind < kKinds; ++kind) {
        if (h[kind]) rc = 1;
        printf("kind %d: %llu differ\n", kind, h[kind]);
    }
    return rc;
}
"""


def test_integer_sum_equals_the_fp64_additions(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src, exe = tmp_path / "sum6.cu", tmp_path / "sum6"
    src.write_text(PROBE)
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O3", "--fmad=false",
                    "-I", os.path.join(REPO, "nyx_gb300", "csrc"), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
