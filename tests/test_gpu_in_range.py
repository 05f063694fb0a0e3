"""The in-range square root and quotients of csrc/mp_dev.cuh against sqrtf and /
on the device, on every float of the ranges that their comments state (for the
division by h^2: every significand, for the cell sizes 1/4 ... 1/512 and some
that are no reciprocals). The check is compiled from the header with the
library's flags."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SRC = r"""
#include <cstdio>
#include <cstring>
#include "mp_dev.cuh"
using namespace mpk;
enum { SQRT, QUOT, SLOPE, THIRD, BY_H2 };
__device__ bool differ(float a, float b) { return __float_as_uint(a) != __float_as_uint(b); }
__global__ void check(int what, uint32_t lo, uint32_t hi, CgQuot c, unsigned long long* bad) {
    unsigned long long n = 0;
    for (uint64_t u = lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u <= hi; u += (uint64_t)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((uint32_t)u), a = 1.4f * 1.4f;
        switch (what) {
        case SQRT: n += differ(sqrt_in_range(x), sqrtf(x)); break;
        case QUOT: n += differ(quot_in_range(a, x), a / x); break;
        case SLOPE: { const float q = a / x; n += differ(quot_in_range(q, x), q / x); break; }
        case THIRD: n += differ(third(x), x / 3.0f) + differ(third(-x), -x / 3.0f) + differ(third(0.0f), 0.0f); break;
        default: n += differ(cg_quot(x, c), x / c.hf) + differ(cg_quot(-x, c), -x / c.hf);
        }
    }
    if (n) atomicAdd(bad, n);
}
// pseudo-random doubles (splitmix64) of magnitude 2^-200 to 2^200
__global__ void check64(CgQuot c, uint64_t seed, unsigned long long* bad) {
    uint64_t z = seed + 0x9e3779b97f4a7c15ull * ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x + 1);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull; z = (z ^ (z >> 27)) * 0x94d049bb133111ebull; z ^= z >> 31;
    const uint64_t e = 1023 - 200 + (z >> 52) % 400;
    const double x = __longlong_as_double((long long)((e << 52) | (z & 0xfffffffffffffull)));
    if (cg_quot(x, c) != x / c.hd) atomicAdd(bad, 1ull);
}
static uint32_t bits(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
static CgQuot quot(float h) {
    CgQuot c;
    c.hf = h * h; c.hd = (double)h * (double)h;
    c.f = 1.0f / c.hf; c.d = 1.0 / c.hd;
    return c;
}
int main() {
    unsigned long long *bad, n = 0;
    cudaMallocManaged(&bad, sizeof(*bad));
    auto run = [&](const char* name, int what, float lo, float hi, CgQuot c = CgQuot()) {
        *bad = 0;
        check<<<148 * 8, 256>>>(what, bits(lo), bits(hi), c, bad);
        if (cudaDeviceSynchronize() != cudaSuccess) { printf("error\n"); return; }
        if (name) printf("%s %llu\n", name, *bad);
        n += *bad;
    };
    run("sqrt", SQRT, 0x1p-100f, 0x1p100f);
    run("quot", QUOT, 0x1p-100f, 0x1p100f);
    run("slope", SLOPE, 1e-4f, 1.96f);
    run("third", THIRD, 0x1p-100f, 0x1p100f);
    n = 0;
    for (int k = 4; k <= 512; k++) run(nullptr, BY_H2, 1.0f, 0x1.fffffep0f, quot(1.0f / k));
    for (float h : {0.013f, 0.1f, 0.37f, 1.7f, 33.0f}) run(nullptr, BY_H2, 1.0f, 0x1.fffffep0f, quot(h));
    printf("by_h2 %llu\n", n);
    n = 0;
    run(nullptr, BY_H2, 4e-31f, 0x1p100f, quot(1.0f / 90));      // the whole range for two
    run(nullptr, BY_H2, 4e-31f, 0x1p100f, quot(1.0f / 200));
    printf("by_h2_range %llu\n", n);
    *bad = 0;
    for (int k = 4; k <= 512; k++) check64<<<148 * 8, 256>>>(quot(1.0f / k), 1000003ull * k, bad);
    if (cudaDeviceSynchronize() != cudaSuccess) { printf("error\n"); return 1; }
    printf("by_h2_double %llu\n", *bad);
    return 0;
}
"""


def test_every_float_of_the_ranges(tmp_path):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "in_range.cu", tmp_path / "in_range"
    src.write_text(SRC)
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false", "-ccbin",
                        "/usr/bin/g++", "-I", os.path.join(ROOT, "2017multiphase_b200", "csrc"), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    counts = dict(line.split() for line in r.stdout.splitlines())
    assert counts == {k: "0" for k in ("sqrt", "quot", "slope", "third", "by_h2", "by_h2_range", "by_h2_double")}
