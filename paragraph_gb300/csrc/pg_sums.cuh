// pg_sums.cuh -- short sums of fp32 values and products to 64-bit accuracy in fp32 arithmetic, host and
// device.
#pragma once
#include "pg_core.cuh"

namespace pg {

// a + b = s + err exactly (Knuth's two-sum; the build neither contracts nor reassociates)
PG_HD float two_sum(float a, float b, float& err) {
    const float s = a + b;
    const float bb = s - a;
    err = (a - (s - bb)) + (b - bb);
    return s;
}

// A sum of at most 32 fp32 values or products.  s carries the sum, e the rounding errors of s (and of the
// products, exact by FMA), t the rounding errors of e: what is lost are the roundings of t, 2^-24 of 2^-24 of
// an error, below 2^-60 of the terms' magnitudes, so the value is the exact sum up to its own 64-bit rounding.
// GB300 does two FP64 operations per clock and SM against 128 in fp32.  It holds while no sum or product
// overflows and no product's error underflows: err_ranges_hold says so for a sum of weights w (not negative)
// and the products w f beside it with |f| up to 2^31 and, unless 0, from 2^-24.
struct ErrSum {
    float s = 0.0f, e = 0.0f, t = 0.0f;
};
PG_HD void err_add(ErrSum& S, float v) {
    float r, q;
    S.s = two_sum(S.s, v, r);
    S.e = two_sum(S.e, r, q);
    S.t += q;
}
PG_HD void err_add_product(ErrSum& S, float a, float b) {
    const float p = a * b, q = fmaf_(a, b, -p);
    float r, u, v;
    S.s = two_sum(S.s, p, r);
    S.e = two_sum(S.e, r, u);
    S.e = two_sum(S.e, q, v);
    S.t += u + v;
}
PG_HD double err_value(const ErrSum& S) { return (double)S.s + ((double)S.e + (double)S.t); }
// products and their sums stay below 2^90 2^31 2^5; a product that matters beside 2^-60 has its error above the
// smallest fp32.  All weights 0 is exact too.
PG_HD bool err_ranges_hold(const ErrSum& S) { return S.s == 0.0f || (S.s >= 0x1p-60f && S.s <= 0x1p90f); }

}  // namespace pg
