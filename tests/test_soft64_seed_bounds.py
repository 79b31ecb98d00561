"""The seeds of csrc/tg_soft64.cuh's reciprocal, quotient and root: on the
host, equal bits with seeds as far off as the correction is said to allow; on
the device, every seed against the error that is claimed for it, and the four
operations against the device's own IEEE ones."""

import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tupan_gb300", "csrc")

HOST = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
// the operand behind a seed (its significand, not truncated) and the error
// wanted: 1 - x r of the reciprocal, 1 - w t^2 of the root
static double operand;
static double wanted;
static bool squared;
static float seed()
{
    const double exact = squared ? sqrt((1.0 - wanted) / operand)
                                 : (1.0 - wanted) / operand;
    float y = (float)exact;
    // the next one inwards, if rounding went past the bound
    const double e = squared ? 1.0 - operand * ((double)y * y)
                             : 1.0 - operand * (double)y;
    if (fabs(e) > fabs(wanted)) y = nextafterf(y, wanted > 0 ? 2.0f : 0.0f);
    return y > 1.0f ? 1.0f : y;
}
#define TG_HOST_SEED(y) ((void)(y), seed())
#include "tg_soft64.cuh"
using namespace tg::soft;
static uint64_t st = 88172645463325252ull;
static uint64_t rnd()
{
    st ^= st << 13; st ^= st >> 7; st ^= st << 17;
    return st * 2685821657736338717ull;
}
static double value()
{
    uint64_t s;
    switch (rnd() % 8) {
    case 0: s = rnd() >> (12 + rnd() % 52); break;
    case 1: s = ~(rnd() >> (12 + rnd() % 52)); break;
    case 2: s = rnd() << (rnd() % 52); break;
    case 3: s = 1ull << (rnd() % 52); break;
    default: s = rnd();
    }
    const uint64_t u = (s & ((1ull << 52) - 1)) |
                       ((523 + rnd() % 1000) << 52) | (rnd() << 63);
    double d;
    memcpy(&d, &u, 8);
    return d;
}
static double significand(double a, bool pair)      // [1, 2), or [1, 4)
{
    int e;
    const double m = 2.0 * frexp(fabs(a), &e);      // a = m 2^(e - 1)
    return pair && !(e & 1) ? 2.0 * m : m;
}
static int differ(double a, double b) { return memcmp(&a, &b, 8) != 0; }
int main(int, char **argv)
{
    const char op = argv[1][0];
    squared = op == 's';
    const double limit = squared ? exp2(-21.2) : exp2(-21.0);
    long bad = 0;
    double most = 0.0;
    for (long k = 0; k < 4000000; ++k) {
        const double a = value(), b = value(), s = fabs(a);
        // at the limit, or anywhere below it
        wanted = limit * (k % 3 ? 1.0 : (double)(rnd() >> 11) / (1ull << 53));
        if (rnd() & 1) wanted = -wanted;
        operand = significand(op == 'q' ? b : a, squared);
        const double y = seed();
        const double e = fabs(squared ? 1.0 - operand * (y * y)
                                      : 1.0 - operand * y);
        if (e > most) most = e;
        if (op == 'r') bad += differ(rcp(s), 1.0 / s);
        if (op == 'q') bad += differ(quo(a, b), a / b);
        if (op == 's') bad += differ(root(s), sqrt(s));
    }
    printf("%ld %d\n", bad, most > 0.95 * limit && most <= limit);
    return 0;
}
"""


@pytest.mark.parametrize("op", ["rcp", "quo", "sqrt"])
def test_bits_with_the_seed_as_far_off_as_allowed(op, tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(HOST)
    subprocess.check_call([cxx, "-O2", "-ffp-contract=off", "-I", CSRC,
                           str(src), "-o", str(exe)])
    # no differences; the limit was come within 5 % of
    assert subprocess.check_output([str(exe), op[0]]).split() == [b"0", b"1"]


DEVICE = r"""
#include <cuda_runtime.h>
#include <math.h>
#include "tg_soft64.cuh"
using namespace tg::soft;
struct Found {
    unsigned long long rcp, rsq;      // largest errors, bits of a double
    unsigned long long bad[4];        // results that differ
};
__device__ void most(unsigned long long *at, double e)
{
    atomicMax(at, (unsigned long long)__double_as_longlong(fabs(e)));
}
// every operand of the seeds: 2^23 in [1, 2), 2^24 in [1, 4), each standing
// for the operands up to the next
__global__ void seeds(Found *f)
{
    const unsigned n = blockIdx.x * blockDim.x + threadIdx.x;
    const double ulp = 1.0 / 8388608.0;
    if (n < (1u << 23)) {
        const float x = as_float(0x3f800000u | n);
        const double r = (double)to_u32(seed_rcp(x) * 2147483648.0f) /
                         2147483648.0;
        most(&f->rcp, fma(-(double)x, r, 1.0));
        most(&f->rcp, fma(-((double)x + ulp), r, 1.0));
    }
    if (n < (1u << 24)) {
        const float w = as_float(0x3f800000u + n);
        const double t = (double)to_u32(seed_rsq(w) * 2147483648.0f) /
                         2147483648.0;
        const double up = (double)w + (w < 2.0f ? ulp : 2.0 * ulp);
        most(&f->rsq, fma(-(double)w, t * t, 1.0));
        most(&f->rsq, fma(-up, t * t, 1.0));
    }
}
__device__ unsigned long long mix(unsigned long long z)
{
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__device__ double value(unsigned long long n)
{
    const unsigned long long a = mix(2 * n), b = mix(2 * n + 1);
    unsigned long long s = a;
    const int sh = (int)((b >> 40) % 52);
    switch ((int)(b >> 60) & 7) {
    case 0: s = a >> (12 + sh); break;
    case 1: s = ~(a >> (12 + sh)); break;
    case 2: s = a << sh; break;
    case 3: s = 1ull << sh; break;
    }
    return __longlong_as_double((long long)(
        (s & ((1ull << 52) - 1)) | ((523ull + (b & 0xffffff) % 1000) << 52) |
        (b & (1ull << 39) ? 1ull << 63 : 0)));
}
__device__ int differ(double a, double b)
{
    return __double_as_longlong(a) != __double_as_longlong(b);
}
__global__ void operations(Found *f, unsigned long long runs)
{
    unsigned long long bad[4] = {0, 0, 0, 0};
    const unsigned long long id =
        (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (unsigned long long k = 0; k < runs; ++k) {
        const double a = value(2 * (id * runs + k)),
                     b = value(2 * (id * runs + k) + 1), s = fabs(a);
        bad[0] += differ(mul(a, b), __dmul_rn(a, b));
        bad[1] += differ(rcp(s), __drcp_rn(s));
        bad[2] += differ(quo(a, b), __ddiv_rn(a, b));
        bad[3] += differ(root(s), __dsqrt_rn(s));
    }
    for (int c = 0; c < 4; ++c)
        if (bad[c]) atomicAdd(&f->bad[c], bad[c]);
}
extern "C" int run(double *errors, unsigned long long *bad)
{
    Found *d, h;
    if (cudaMalloc((void **)&d, sizeof(h)) != cudaSuccess) return 1;
    cudaMemset(d, 0, sizeof(h));
    seeds<<<(1 << 24) / 256, 256>>>(d);
    operations<<<152 * 8, 256>>>(d, 256);
    const cudaError_t e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return 2;
    memcpy(&errors[0], &h.rcp, 8);
    memcpy(&errors[1], &h.rsq, 8);
    for (int c = 0; c < 4; ++c) bad[c] = h.bad[c];
    return 0;
}
"""


@pytest.mark.gpu
def test_every_seed_and_the_device_operations(tmp_path):
    from tupan_gb300 import build
    src, so = tmp_path / "t.cu", tmp_path / "t.so"
    src.write_text("#include <string.h>\n" + DEVICE)
    subprocess.check_call([build.nvcc()] + build.ARCH +
                          ["-O3", "-std=c++17", "-fmad=false", "-I", CSRC,
                           "-shared", "-Xcompiler", "-fPIC", str(src), "-o",
                           str(so)])
    errors = (ctypes.c_double * 2)()
    bad = (ctypes.c_ulonglong * 4)()
    assert ctypes.CDLL(str(so)).run(errors, bad) == 0
    # the seeds' errors: 2^-22.4 of r, 2^-22.5 of t (1 - w t^2 has twice
    # that), inside the 2^-21 and 2^-21.2 that the correction allows
    assert 0.0 < errors[0] <= 2.0 ** -22.4
    assert 0.0 < errors[1] <= 2.0 ** -21.5
    # 80 million operands of each operation
    assert list(bad) == [0, 0, 0, 0]
