// radius_weight.cuh -- the radius gather's weight, w * (1 - s) / exposure in
// double precision rounded to float once, from single-precision arithmetic:
// the same bits for every argument.
//
// 1 - s, its product with 1 / exposure and the product with w are kept as
// unevaluated sums of two floats (Dekker 1971), off by at most 2^-45 of the
// value. The sum rounds to the same float as the double expression unless it
// lies within that error of the middle between two floats, and it overflows,
// or loses its low part to underflow, only where the double expression does
// not: in both cases the double expression is evaluated itself. Moving the low
// part by 2^-16 of itself moves a sum near a middle (half an ulp, or a quarter
// beside a power of two, from r) by 2^-18 ulp at least; the error is 2^-21 ulp
// at most. About one weight in 50,000 is evaluated twice.
#pragma once
#include "pm_vec.cuh"

namespace pm {

PM_HD float radius_weight_double(float w, float s, float exposure) {
    return (float)((double)w * ((1.0 - (double)s) / (double)exposure));
}

// 1 / exposure as a float and the float nearest to the rest. NaN, which sends
// every weight to the double expression, where the rest would lose bits to
// underflow or the float overflows.
PM_HD void radius_inverse(float exposure, float *hi, float *lo) {
    const double r = 1.0 / (double)exposure, a = r < 0.0 ? -r : r;
    const bool fits = a > 1e-28 && a < 1e38;
    *hi = fits ? (float)r : (float)(0.0 / 0.0);
    *lo = fits ? (float)(r - (double)*hi) : 0.0f;
}

PM_HD float radius_weight(float w, float s, float exposure, float hi, float lo) {
    // 1 - s exactly: u + ul
    const float u = 1.0f - s;
    const float bb = u - 1.0f;
    const float ul = (1.0f - (u - bb)) + (-s - bb);
    // times 1 / exposure: p + pl
    const float p = u * hi;
    const float pl = PM_FMAF(u, hi, -p) + PM_FMAF(u, lo, ul * hi);
    // times w: r + e
    const float r = w * p;
    const float e = PM_FMAF(w, p, -r) + w * pl;
    const float up = r + e * 1.0000152587890625f, down = r + e * 0.9999847412109375f;
    const float size = r < 0.0f ? -r : r;
    if (up == down && size > 1e-30f) return up;  // NaN fails the first comparison
    if (w == 0.0f && size == 0.0f) return r;     // a record that faces away: zero with p's sign
    return radius_weight_double(w, s, exposure);
}

}  // namespace pm
