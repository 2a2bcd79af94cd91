// FloatSumOf (kpt_sum.h) with denormals flushed to zero, as the gradient
// kernels run it, against the sum in a double-double (106 bits).  Errors are
// relative to the largest partial sum.
// Prints per size of the terms "<log2> <relative error of the three floats> <of a double>".
#include <cstdint>
#include <cstdio>
#include <algorithm>

#include "kpt_sum.h"

static float flush(float x) { return std::fabs(x) < 0x1p-126f ? 0.0f : x; }
struct Flushed {
    static float add(float a, float b) { return flush(a + b); }
    static float sub(float a, float b) { return flush(a - b); }
    static float mul(float a, float b) { return flush(a * b); }
};

int main() {
    uint64_t state = 1;
    auto draw = [&] { state = state * 6364136223846793005ull + 1442695040888963407ull; return (double)(state >> 11) * 0x1p-53; };
    for (int size : {-120, -110, -100, -90, -80, -70, -40, 0, 40, 80, 92, 98, 104, 120}) {
        double worst = 0.0, worst_double = 0.0;
        for (int trial = 0; trial < 500; ++trial) {
            kpt::FloatSumOf<Flushed> sum;
            double spilled = 0.0, plain = 0.0, largest = 0.0;
            double exact = 0.0, rest = 0.0;   // a double-double
            for (int k = 0; k < 200; ++k) {
                // of both signs, over 40 powers of two
                const float v = flush((float)std::ldexp(draw() - 0.4, size - (int)(40.0 * draw())));
                sum.add(v, [&](double x) { spilled += x; });
                plain += v;
                const double s = exact + v, t = s - exact;
                rest += (exact - (s - t)) + (v - t);
                exact = s;
                largest = std::max(largest, std::fabs(exact));
            }
            const double total = exact + rest;
            const double got = spilled + sum.value();
            worst = std::max(worst, std::fabs(((got - exact) - rest) / largest));
            worst_double = std::max(worst_double, std::fabs((plain - total) / largest));
        }
        std::printf("%d %.3e %.3e\n", size, worst, worst_double);
    }
    return 0;
}
