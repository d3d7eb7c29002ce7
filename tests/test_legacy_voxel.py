"""The legacy mapper's single-precision conversions (csrc/legacy_voxel.cuh)
against the double expressions they stand for, on the CPU: every float
within 64 ulp of a step, both signs around zero, a stride over all float
bit patterns, infinities and NaN. Equal integers and bytes throughout."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <math.h>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include "legacy_voxel.cuh"
using namespace pm;
static float bits(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static long bad = 0;
static void check(float x) {
    const float l = 1.0f - x, d = (float)(1.0 - (double)x);
    const bool ok = legacy_voxel_xy(x) == legacy_voxel_xy_general(x) && legacy_voxel_z(x) == legacy_voxel_z_general(x) &&
                    unit_to_u8(x) == to_u8_sat((double)x * 255.0) && (memcmp(&l, &d, 4) == 0 || (l != l && d != d)) &&
                    (x < -0.00001f) == ((double)x < -0.00001);
    if (!ok && bad++ < 10) printf("%.9g\n", x);
}
static void around(float x) {
    uint32_t u;
    memcpy(&u, &x, 4);
    for (int i = -64; i <= 64; ++i) { check(bits(u + i)); check(-bits(u + i)); }
}
int main() {
    for (int k = -800; k <= 800; ++k) { around(legacy_step_xy(k)); around(legacy_step_z(k)); }
    for (int i = 0; i <= 256; ++i) around((float)(i / 255.0));
    for (int e = 0; e < 255; ++e) around(bits((uint32_t)e << 23));
    for (float x : {64.0f, 1e9f, 3.4e38f, INFINITY, NAN, 1.1102230246251565e-16f, 0.00001f}) around(x);
    for (uint64_t u = 0; u < (1ull << 32); u += 1009) check(bits((uint32_t)u));
    for (int v = -3000000; v < 3000000; v += 7) {
        if (legacy_world_xy(v) != (float)((double)((float)v / 32.0f) * 3.0 - 1.5)) ++bad;
        if (legacy_world_z(v) != (float)((double)((float)v / 32.0f) * 6.0)) ++bad;
    }
    printf("%ld\n", bad);
    return bad != 0;
}
"""


def test_single_precision_conversions_equal_the_double_ones(tmp_path):
    src = tmp_path / "harness.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "harness"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "cuda-photon-mapper_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert out.returncode == 0, out.stdout
