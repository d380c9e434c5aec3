"""The exact helpers of the FP64 kernel (csrc/stage64.cuh) and the conversions by
integer operations (csrc/split.cuh), bit for bit against the plain operations that
they stand for: random arguments of all magnitudes, and the edges (zeros of both
signs, subnormals, powers of two and their neighbours, the limits of the fast
paths, ties, infinities and NaN), every edge against every other."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>
#include "split.cuh"
#include "stage64.cuh"
using namespace b2d;

enum { DIVIDE, BACK, MINMOD, NARROW, SPLIT, WIDEN, HALVE, COUNT };
static const char* names[] = {"Divisor", "ThereAndBack", "minmod_bits", "narrow", "split_double", "widen", "halve"};

// the same bits, or NaN both
__device__ bool same(double a, double b) { return dbits(a) == dbits(b) || (a != a && b != b); }
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }

__device__ void note(unsigned long long* n, double* first, int what, double a, double b, double c)
{
    if (atomicAdd(n + what, 1ull) == 0ull) {
        first[3 * what] = a;
        first[3 * what + 1] = b;
        first[3 * what + 2] = c;
    }
}

__global__ void check(const double* A, const double* B, const double* C, long long n, unsigned long long* bad, double* first)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double a = A[i], b = B[i], c = C[i];
        if (!same(Divisor(b)(a), plain_div(a, b))) note(bad, first, DIVIDE, a, b, 0.0);
        if (!same(ThereAndBack(b)(a), plain_div(a * b, b))) note(bad, first, BACK, a, b, 0.0);
        const double m = minmod_bits(a, b, c), want = minmod_nan(a, 0.5 * b, c);
        if (!(m == want || (m != m && want != want))) note(bad, first, MINMOD, a, b, c);   // (the sign of a zero does not matter)
        if (!same(narrow(a), (float)a)) note(bad, first, NARROW, a, 0.0, 0.0);
        float hi, lo;
        split_double(a, hi, lo);
        const float wlo = (float)(a - (double)hi);
        if (!same(hi, (float)a) || !(lo == wlo || (lo != lo && wlo != wlo))) note(bad, first, SPLIT, a, hi, lo);
        const float f = (float)a;
        if (!same(widen(f), (double)f)) note(bad, first, WIDEN, a, 0.0, 0.0);
        if (!same(halve(a), 0.5 * a)) note(bad, first, HALVE, a, 0.0, 0.0);
    }
}

int main()
{
    std::vector<double> edges;
    auto around = [&](double v) {
        for (double s : {v, -v})
            for (double w : {s, std::nextafter(s, 0.0), std::nextafter(s, 2.0 * s)}) edges.push_back(w);
    };
    for (int e : {-1073, -1022, -1021, -1000, -401, -400, -399, -149, -126, -125, -71, -70, -69, -26, -25, -24, -23, -2, -1,
                  0, 1, 2, 23, 24, 25, 52, 53, 99, 100, 101, 126, 127, 128, 398, 399, 400, 401, 1000, 1022, 1023})
        around(std::ldexp(1.0, e));
    for (int k = 0; k < 8; ++k) {   // ties of the 24-bit rounding, and a bit beside them
        around(1.0 + std::ldexp((double)k, -24));
        around(std::ldexp(2.0 - std::ldexp((double)k, -25), 30));
    }
    for (double v : {3.0, 1.0 / 3.0, 10.0, 0.1}) around(v);
    const double inf = std::numeric_limits<double>::infinity();
    for (double v : {0.0, -0.0, inf, -inf, std::numeric_limits<double>::quiet_NaN(), std::numeric_limits<double>::max()}) edges.push_back(v);
    std::vector<double> a, b, c;
    for (size_t i = 0; i < edges.size(); ++i)
        for (size_t j = 0; j < edges.size(); ++j) {
            a.push_back(edges[i]);
            b.push_back(edges[j]);
            c.push_back(edges[(i * 7 + j * 13) % edges.size()]);
        }
    std::mt19937_64 rng(12345);
    auto random = [&](int lo, int hi) {
        const unsigned long long m = rng();
        unsigned long long w = (m >> 12) | ((unsigned long long)(1023 + lo + (int)(rng() % (unsigned)(hi - lo + 1))) << 52) | (m << 63);
        if (rng() % 8 == 0) w &= ~((1ull << (rng() % 52)) - 1);   // few bits
        double v;
        memcpy(&v, &w, 8);
        return v;
    };
    for (int i = 0; i < 6000000; ++i) {
        const int range = i % 3 == 0 ? 3 : i % 3 == 1 ? 80 : 420;
        a.push_back(random(-range, range));
        b.push_back(random(-range, range));
        c.push_back(random(-range, range));
    }
    const long long n = (long long)a.size();
    double *d[3], *first;
    unsigned long long* bad;
    for (int k = 0; k < 3; ++k) {
        cudaMalloc(&d[k], 8 * n);
        cudaMemcpy(d[k], (k == 0 ? a : k == 1 ? b : c).data(), 8 * n, cudaMemcpyHostToDevice);
    }
    cudaMalloc(&bad, 8 * COUNT);
    cudaMalloc(&first, 24 * COUNT);
    cudaMemset(bad, 0, 8 * COUNT);
    check<<<608, 256>>>(d[0], d[1], d[2], n, bad, first);
    unsigned long long h[COUNT];
    double f[3 * COUNT];
    if (cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) {
        printf("%s\n", cudaGetErrorString(cudaGetLastError()));
        return 2;
    }
    cudaMemcpy(f, first, sizeof f, cudaMemcpyDeviceToHost);
    int rc = 0;
    for (int k = 0; k < COUNT; ++k)
        if (h[k]) {
            printf("%s: %llu of %lld differ, one at %a %a %a\n", names[k], h[k], n, f[3 * k], f[3 * k + 1], f[3 * k + 2]);
            rc = 1;
        }
    return rc;
}
"""


@pytest.mark.parametrize("flags", [["--fmad=false"], ["--fmad=false", "-ftz=true"]], ids=["plain", "ftz"])
def test_helpers_equal_the_operations(tmp_path, flags):
    """With the flags of the units that use them (the FP32 units flush subnormals)."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "helpers.cu", tmp_path / "helpers"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", *flags, "-I",
                    os.path.join(ROOT, "app-binary2d_gb300", "csrc"), "-I", os.path.join(ROOT, "include"), str(src), "-o",
                    str(exe)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
