"""The radius gather's single-precision weight (csrc/radius_weight.cuh) is the
double expression's, bit for bit: random and edge weights, distances and
exposures over the whole float range, and arguments beside the middle between
two floats, on the CPU."""
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
static long bad = 0;
static void check(float w, float s, float e) {
    float hi, lo;
    radius_inverse(e, &hi, &lo);
    const float a = radius_weight(w, s, e, hi, lo), b = radius_weight_double(w, s, e);
    if (memcmp(&a, &b, 4) != 0 && !(a != a && b != b) && bad++ < 10)
        printf("w %.9g s %.9g exposure %.9g: %.9g, not %.9g\n", w, s, e, a, b);
}
int main() {
    const float edge[] = {0.0f, 1.0f, 0.5f, 0x1p-24f, 0x1p-25f, 1.0f - 0x1p-24f, 1.0f + 0x1p-23f, 3.0f, 1e9f, 1e19f,
                          3.4e38f, 1e-20f, 1e-38f, 1e-45f, INFINITY, NAN};
    const float expo[] = {50.0f, 1.0f, -2.0f, 3.0f, 3e-7f, 1e15f, 5e25f, 1e-32f, 2e-30f, 1e-38f, 1e-45f, 3e38f, 7e27f,
                          1e28f, INFINITY, NAN};
    for (float w : edge) for (float s : edge) for (float e : expo) { check(w, s, e); check(w, s, -e); }
    for (long i = 0; i < 8000000; ++i) check(unit(), sqrtf(unit()), 50.0f);
    for (long i = 0; i < 3000000; ++i) check(unit(), 2.0f * unit(), bits(0x30000000u + (rnd() & 0x1fffffffu)));
    for (long i = 0; i < 3000000; ++i) check(fabsf(bits(rnd())), fabsf(bits(rnd())), bits(rnd()));
    // products that lie on, or one part in 2^52 beside, the middle between two floats
    for (long i = 0; i < 1000000; ++i) {
        const float s = (float)(int)(rnd() & 1023u) * 0x1p-10f, w = 1.0f + (float)(int)(rnd() & 0x7fffu) * 0x1p-15f;
        check(w, s, 1.0f);
        check(w, s, 0.25f);
        check(w * 0x1p-3f, s, 3.0f);
        check(w, bits(0x3f000000u + (rnd() & 0xffu)), 1.0f + 0x1p-23f * (float)(rnd() & 7u));
    }
    printf("%ld\n", bad);
    return bad != 0;
}
"""


def test_weight_is_the_double_expression(tmp_path):
    src = tmp_path / "harness.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "harness"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "cuda-photon-mapper_gb300", "csrc"), str(src), "-o", str(exe), "-lm"], check=True)
    out = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert out.returncode == 0, out.stdout
