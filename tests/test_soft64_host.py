"""The integer-pipe product, reciprocal, quotient and root of
csrc/tg_soft64.cuh, compiled for the host, against the host's IEEE ones:
equal bits over structured and random significands, with the seeds shifted
by up to the error the device's approximations have."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
static int shift = 0;
// `shift` units of 2^-24 relative to 1: a seed in [1/2, 1]
static inline float moved(float y)
{
    float z = y + shift * y * 5.9604645e-8f;
    return z > 1.0f ? 1.0f : z;
}
#define TG_HOST_SEED(y) moved(y)
#include "tg_soft64.cuh"
using namespace tg::soft;
static uint64_t st = 88172645463325252ull;
static uint64_t rnd()
{
    st ^= st << 13; st ^= st >> 7; st ^= st << 17;
    return st * 2685821657736338717ull;
}
static uint64_t significand()
{
    switch (rnd() % 8) {
    case 0: return rnd() >> (12 + rnd() % 52);
    case 1: return ~(rnd() >> (12 + rnd() % 52));
    case 2: return rnd() << (rnd() % 52);
    case 3: return 1ull << (rnd() % 52);
    default: return rnd();
    }
}
static double value()
{
    uint64_t u = (significand() & ((1ull << 52) - 1)) |
                 ((523 + rnd() % 1000) << 52) | (rnd() << 63);
    double d;
    memcpy(&d, &u, 8);
    return d;
}
static int differ(double a, double b) { return memcmp(&a, &b, 8) != 0; }
int main(int, char **argv)
{
    const char op = argv[1][0];
    long bad = 0;
    for (long k = 0; k < 4000000; ++k) {
        const double a = value(), b = value(), s = fabs(a);
        shift = (int)(rnd() % 5) - 2;
        if (op == 'm') bad += differ(mul(a, b), a * b);
        if (op == 'r') bad += differ(rcp(s), 1.0 / s);
        if (op == 'q') bad += differ(quo(a, b), a / b);
        if (op == 's') bad += differ(root(s), sqrt(s));
        if (range_key(a) >= RANGE) ++bad;
    }
    const double out[] = {0.0, -0.0, 5e-324, 1e-200, 1e200,
                          strtod("inf", 0), strtod("nan", 0)};
    for (double x : out) bad += range_key(x) < RANGE;
    printf("%ld\n", bad);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("soft64")
    src = d / "t.cpp"
    src.write_text(SOURCE)
    subprocess.check_call([cxx, "-O2", "-ffp-contract=off", "-I",
                           os.path.join(ROOT, "tupan_gb300", "csrc"),
                           str(src), "-o", str(d / "t")])
    return str(d / "t")


@pytest.mark.parametrize("op", ["mul", "rcp", "quo", "sqrt"])
def test_bits_equal_the_ieee_operations(program, op):
    assert subprocess.check_output([program, op[0]]).split() == [b"0"]
