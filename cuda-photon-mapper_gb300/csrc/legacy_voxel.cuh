// legacy_voxel.cuh -- the legacy mapper's double-precision conversions in
// single precision, with the same results for every input.
//
// The reference finds a voxel as the truncation of a double expression
// (getVoxelCoordinates, photonMappingKernel.cu:254-261) ten times per pixel
// and more, each a double division; this GPU runs double precision at a
// small fraction of its single-precision rate. The expression is monotone in
// its float argument and its steps lie at multiples of 1/32 (x, y: 3k/32 -
// 1.5) and 1/16 (z: 3k/16), which are floats, so a single-precision guess
// corrected against the neighbouring steps gives the same integer: a float
// below a step is below it by 2^-24 of its size at least, far more than the
// double expression's rounding. One step of x and y is not at its float:
// 16, at zero, where x + 1.5 already rounds to 1.5 for x from -2^-53 up.
#pragma once
#include "pm_vec.cuh"

namespace pm {

PM_HD int legacy_voxel_xy_general(float x) { return d2i_sat((((double)x + 1.5) / 3.0) * 32.0); }
PM_HD int legacy_voxel_z_general(float z) { return d2i_sat(((double)z / 6.0) * 32.0); }

// Step k of a coordinate, exact for |k| < 2^20.
PM_HD float legacy_step_xy(int k) { return (float)(3 * k - 48) * 0.03125f; }
PM_HD float legacy_step_z(int k) { return (float)(3 * k) * 0.0625f; }

// Coordinates the single-precision steps cover.
constexpr float kLegacyFastRange = 64.0f;

PM_HD int legacy_voxel_xy(float x) {
    if (!(x > -kLegacyFastRange && x < kLegacyFastRange)) return legacy_voxel_xy_general(x);  // and NaN
    int k = (int)PM_FLOORF((x + 1.5f) * 10.6666667f);
    const float at = k == 16 ? -1.1102230246251565e-16f : legacy_step_xy(k);
    const float above = k == 15 ? -1.1102230246251565e-16f : legacy_step_xy(k + 1);
    if (x < at) --k;
    else if (x >= above) ++k;
    // truncation toward zero: below zero a value between steps takes the upper one
    return k < 0 && x != legacy_step_xy(k) ? k + 1 : k;
}

PM_HD int legacy_voxel_z(float z) {
    if (!(z > -kLegacyFastRange && z < kLegacyFastRange)) return legacy_voxel_z_general(z);
    int k = (int)PM_FLOORF(z * 5.33333349f);
    if (z < legacy_step_z(k)) --k;
    else if (z >= legacy_step_z(k + 1)) ++k;
    return k < 0 && z != legacy_step_z(k) ? k + 1 : k;
}

// World coordinates of a voxel's lower corner (getWorldCoordinates,
// :263-268): exact in single precision while three times the index fits its
// significand.
PM_HD float legacy_world_xy(int v) {
    if (v > -(1 << 20) && v < (1 << 20)) return ((float)v / 32.0f) * 3.0f - 1.5f;
    return (float)((double)((float)v / 32.0f) * 3.0 - 1.5);
}
PM_HD float legacy_world_z(int v) {
    if (v > -(1 << 20) && v < (1 << 20)) return ((float)v / 32.0f) * 6.0f;
    return (float)((double)((float)v / 32.0f) * 6.0);
}

}  // namespace pm
