// n64_margin.cpp -- how far the triple-float sqrt, reciprocal and quotient that
// ag::n64 rounds (ag_tf64.cuh) lie from the exact values (__float128), in ulps
// of the exact result's double. Prints one JSON object of the largest
// distances over a seeded corpus. Test infrastructure.
#include "host_shim.h"

#include <quadmath.h>

#include <cstdio>
#include <cstring>
#include <random>

inline double __dmul_rn(double a, double b) { return a * b; }
inline int __float2int_rn(float f) { return (int)std::nearbyintf(f); }
namespace ag {
namespace n64 {
inline double slow_sqrt(double x) { return std::sqrt(x); }
inline double slow_rsqrt(double x) { return 1.0 / std::sqrt(x); }
inline double slow_div(double a, double b) { return a / b; }
inline double slow_exp(double x) { return std::exp(x); }
inline double slow_log(double x) { return std::log(x); }
inline double slow_log1p(double x) { return std::log1p(x); }
}  // namespace n64
}  // namespace ag
#define AG_N64_HOST_CHECK
#include "../../include/aether/gb300/ag_tf64.cuh"

typedef __float128 Q;
static double far(ag::t64::tf v, Q ref) {
    int e;
    frexpq(fabsq(ref), &e);
    return (double)(fabsq((Q)v.x + v.y + v.z - ref) / ldexpq((Q)1, e - 53));
}

int main() {
    using namespace ag;
    std::mt19937_64 rng(5);
    // all significands, and ones near 1 and 2
    auto draw = [&] {
        const uint64_t b = (rng() >> 12) | 0x3ff0000000000000ull;
        double d;
        std::memcpy(&d, &b, 8);
        const int k = int(rng() % 8), s = int(rng() % 50);
        if (k == 0) d = 1.0 + std::ldexp(d - 1.0, -s);
        if (k == 1) d = 2.0 - std::ldexp(d - 1.0, -s);
        return std::ldexp(d, int(rng() % 60) - 30);
    };
    double root = 0, inverse = 0, quotient = 0;
    for (int i = 0; i < 300000; ++i) {
        bool ok = true;
        const double x = draw(), y = (rng() & 1 ? 1.0 : -1.0) * draw();
        const t64::tf a = n64::split(x, ok), b = n64::split(y, ok), r = t64::recip(b);
        root = std::fmax(root, far(t64::sqrt_pos_(a), sqrtq((Q)x)));
        inverse = std::fmax(inverse, far(r, 1 / (Q)y));
        quotient = std::fmax(quotient, far(t64::mul(a, r), (Q)x / (Q)y));
    }
    std::printf("{\"sqrt\": %.9f, \"recip\": %.9f, \"div\": %.9f}\n", root, inverse, quotient);
}
