// kpt_sum.h -- sums of many floats, also as plain C++ (tests/float_sum.cpp
// checks them on the CPU).
#pragma once

#ifdef __CUDACC__
#define KPT_SUM_FN __device__ __forceinline__
#else
#include <cmath>
#define KPT_SUM_FN inline
#endif

namespace kpt {

// A sum of floats as three floats: each addition's rounding error is kept in
// the next (two-sums), the last of them good to 2^-72 of the largest partial
// sum -- nearer than a double, whose additions run at 1/64 of the float rate.
// The floats hold 2^24 times the sum: a term is 0 or a multiple of 2^-149 (its
// denormals are zero), so every rounding error is 0 or at least 2^-125, and
// none is lost where denormals are flushed.  (Unscaled, 200 terms of up
// to 2^-100 were summed to 4e-7.)  A sum that leaves 2^100, or infinity or NaN, goes to
// spill(double).  Arith: add, sub, mul, one rounding each.
template <class Arith>
struct FloatSumOf {
    float hi = 0.0f, mid = 0.0f, lo = 0.0f;
    static KPT_SUM_FN float two_sum(float& a, float b) {   // a += b, returning the error
        const float s = Arith::add(a, b), t = Arith::sub(s, a);
        const float e = Arith::add(Arith::sub(a, Arith::sub(s, t)), Arith::sub(b, t));
        a = s;
        return e;
    }
    KPT_SUM_FN double value() const { return ((double)hi + ((double)mid + (double)lo)) * 0x1p-24; }
    template <class Spill>
    KPT_SUM_FN void add(float v, Spill spill) {
        const float w = Arith::mul(v, 0x1p24f);
        if (fabsf(Arith::add(hi, w)) < 0x1p124f) {
            float e = two_sum(hi, w);
            e = two_sum(mid, e);
            lo = Arith::add(lo, e);
        } else {
            spill(value() + (double)v);
            hi = mid = lo = 0.0f;
        }
    }
};

}  // namespace kpt
