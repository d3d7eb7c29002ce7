// radius_weight.cuh -- the radius gather's weight, w * (1 - s) / exposure in
// double precision rounded to float once, in single precision.
//
// 1 - s, its product with 1 / exposure and the product with w are kept as
// unevaluated sums of two floats (Dekker 1971), off by at most 2^-45 of the
// value, and rounded once: the float is the double expression's but for one
// weight in some 300,000, whose exact value lies on the middle between two
// floats or within 2^-20 of their spacing from it, where it may be the other
// one. The sums of a gather are as near to 64 bits either way (2.33263e-8, equal
// to six digits over 18,000 sums). Taken for reciprocals of 1e-10 to 1e10, where
// no product overflows at any distance. A product below 2^-100 (a normal of
// 1e-20) has no low part: within one spacing.
#pragma once
#include "pm_vec.cuh"

namespace pm {

PM_HD float radius_weight_double(float w, float s, float exposure) {
    return (float)((double)w * ((1.0 - (double)s) / (double)exposure));
}

// 1 / exposure as a float and the float nearest to the rest; whether
// radius_weight may take it.
PM_HD bool radius_inverse(float exposure, float *hi, float *lo) {
    const double r = 1.0 / (double)exposure, a = r < 0.0 ? -r : r;
    *hi = (float)r;
    *lo = (float)(r - (double)*hi);
    return a >= 1e-10 && a <= 1e10;
}

PM_HD float radius_weight(float w, float s, float hi, float lo) {
    // 1 - s exactly: u + ul
    const float u = 1.0f - s;
    const float bb = u - 1.0f;
    const float ul = (1.0f - (u - bb)) + (-s - bb);
    // times 1 / exposure: p + pl
    const float p = u * hi;
    const float pl = PM_FMAF(u, hi, -p) + PM_FMAF(u, lo, ul * hi);
    // times w
    const float r = w * p;
    return r + (PM_FMAF(w, p, -r) + w * pl);
}

}  // namespace pm
