"""The radius gather's weight as pairs of floats (csrc/radius_weight.cuh)
against the double expression, on the CPU, over every distance and over the
exposures and weights that the pairs are taken for: the same float, or the
other of two that are equally near, but for one in a million (an error of 2^-45
of the value, 2^-21 of a spacing to either side), and then never further from the
exact value than half a spacing and 2^-20 of it."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include "radius_weight.cuh"
using namespace pm;
static uint64_t st = 88172645463325252ull;
static uint32_t rnd() { st ^= st << 13; st ^= st >> 7; st ^= st << 17; return (uint32_t)(st >> 16); }
static float bits(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static float unit() { return (rnd() >> 8) * 0x1p-24f; }
static long bad = 0, other = 0, all = 0;
static void check(float w, float s, float e) {
    float hi, lo;
    if (!radius_inverse(e, &hi, &lo)) { ++bad; return; }
    const float a = radius_weight(w, s, hi, lo), b = radius_weight_double(w, s, e);
    ++all;
    if (a == b) return;  // zeros of either sign are equal
    // the exact value in 64 bits of significand: w (1 - s) is exact to 2^-64 of it
    const long double x = (long double)w * (1.0L - (long double)s) / (long double)e;
    if (fabsl((long double)a - x) != fabsl((long double)b - x)) ++other;
    const float n = nextafterf(a, b);
    const long double spacing = fabsl((long double)b - (long double)a);
    if (n != b || fabsl((long double)a - x) > spacing * (0.5L + 0x1p-20L)) {
        if (bad++ < 10) printf("w %.9g s %.9g exposure %.9g: %.9g, not %.9g\n", w, s, e, a, b);
    }
}
static float expo() { return ldexpf(1.0f + unit(), (int)(rnd() % 65u) - 32) * (rnd() & 1 ? 1.0f : -1.0f); }
int main() {
    const float ws[] = {0.0f, 1.0f, 0.5f, 0x1p-24f, 1.0f - 0x1p-24f, 1.0f + 0x1p-23f, 1.7f, 1e-18f, 1e6f};
    const float ss[] = {0.0f, 1.0f, 0.5f, 0x1p-24f, 0x1p-25f, 0x1p-60f, 1.0f - 0x1p-24f, 1.0f + 0x1p-23f, 3.0f, 1e9f, 1.8e19f};
    const float es[] = {50.0f, 1.0f, -2.0f, 3.0f, 3e-7f, 1.1e-10f, 0.9e10f, -0.9e10f};
    for (float w : ws) for (float s : ss) for (float e : es) check(w, s, e);
    for (long i = 0; i < 20000000; ++i) check(unit(), sqrtf(unit()), 50.0f);
    for (long i = 0; i < 5000000; ++i) check(unit(), 2.0f * unit(), expo());
    for (long i = 0; i < 5000000; ++i) check(ldexpf(1.0f + unit(), -(int)(rnd() % 60u)), ldexpf(1.0f + unit(), (int)(rnd() % 90u) - 30), expo());
    if (other > all / 1000000) { printf("%ld of %ld are the other neighbour\n", other, all); ++bad; }
    // exact values on the middle between two floats, and beside it
    for (long i = 0; i < 2000000; ++i) {
        const float s = (float)(int)(rnd() & 1023u) * 0x1p-10f, w = 1.0f + (float)(int)(rnd() & 0x7fffu) * 0x1p-15f;
        check(w, s, 1.0f);
        check(w, s, 3.0f);
    }
    printf("%ld\n", bad);
    return bad != 0;
}
"""


def test_weight_against_the_double_expression(tmp_path):
    src = tmp_path / "harness.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "harness"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "cuda-photon-mapper_gb300", "csrc"), str(src), "-o", str(exe), "-lm"], check=True)
    out = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert out.returncode == 0, out.stdout
