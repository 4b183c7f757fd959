// The Newton step of the traversal's reciprocals (reciprocal() in ftb_kernels.cu), from the
// float next to 1 / x on either side and from it, over every mantissa (test infrastructure, run
// by tests/test_reciprocal.py).  A start within 1.5 ulp of 1 / x is off by e <= 1.5 * 2^-23 of
// it, the step without its rounding by e^2 <= 2.25 * 2^-46, which is at most 2.25 * 2^-22 ulp, and
// its one rounding by half an ulp.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>

int main() {
    double worst = 0.0;
    long rounded = 0, total = 0;
    for (uint32_t m = 0; m < (1u << 23); ++m) {
        const uint32_t bits = 127u << 23 | m;
        float x;
        std::memcpy(&x, &bits, sizeof x);
        const double exact = 1.0 / (double)x, ulp = std::ldexp(1.0, std::ilogb(exact) - 23);
        const float near = 1.0f / x;
        for (float r : {std::nextafterf(near, 0.0f), near, std::nextafterf(near, 2.0f)}) {
            const float s = std::fmaf(r, std::fmaf(-x, r, 1.0f), r);
            worst = std::fmax(worst, std::fabs((double)s - exact) / ulp);
            rounded += s == near;
            ++total;
        }
    }
    const bool ok = worst <= 0.5 + 2.25 * std::ldexp(1.0, -22);
    std::printf("worst %.9f ulp, %ld of %ld correctly rounded: %s\n", worst, rounded, total, ok ? "ok" : "wrong");
    return ok ? 0 : 1;
}
