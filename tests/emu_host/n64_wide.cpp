// n64_wide.cpp -- ag::n64's sqrt, rsqrt, div, exp, log and log1p over every
// exponent of a double and on special values, sin and cos up to 2^22 and beyond: results that differ from the
// correctly rounded ones (sqrt, rsqrt, div), the largest error in ulps (the
// others), and how many arguments reached the FP64 function. Prints one JSON
// object. Test infrastructure.
#include "host_shim.h"

#include <quadmath.h>

#include <cstdio>
#include <limits>
#include <random>

inline double __dmul_rn(double a, double b) { return a * b; }
inline int __float2int_rn(float f) {   // saturates, NaN gives 0, as on the device
    if (f != f) return 0;
    if (f >= 2147483648.0f) return 2147483647;
    if (f < -2147483648.0f) return -2147483647 - 1;
    return (int)std::nearbyintf(f);
}
static long g_slow;
namespace ag {
inline double f_exp(double x) { return std::exp(x); }
inline double f_sin(double x) { return std::sin(x); }
inline double f_cos(double x) { return std::cos(x); }
namespace n64 {
inline double slow_sqrt(double x) { ++g_slow; return std::sqrt(x); }
inline double slow_rsqrt(double x) { ++g_slow; return 1.0 / std::sqrt(x); }
inline double slow_div(double a, double b) { ++g_slow; return a / b; }
inline double slow_exp(double x) { ++g_slow; return (double)expq((__float128)x); }
inline double slow_log(double x) { ++g_slow; return (double)logq((__float128)x); }
inline double slow_log1p(double x) { ++g_slow; return (double)log1pq((__float128)x); }
inline double slow_sin(double x) { ++g_slow; return (double)sinq((__float128)x); }
inline double slow_cos(double x) { ++g_slow; return (double)cosq((__float128)x); }
inline double slow_normal(ag_u64 seed, ag_u32 g, ag_u32 c) {
    const q4 x = philox_block(seed, g, c);
    const double u = (double)((ag_u64)x.x ^ ((ag_u64)x.y << 21)) * 0x1p-53 + 0x1p-54;
    const double v = (double)((ag_u64)x.z ^ ((ag_u64)x.w << 21)) * 0x1p-52 + 0x1p-53;
    const double s = std::sqrt(-2.0 * (double)logq((__float128)u));
    return s * (double)sinq((__float128)(v * 3.1415926535897932));
}
}  // namespace n64
}  // namespace ag
#define AG_N64_HOST_CHECK
#include "../../include/aether/gb300/ag_tf64.cuh"
#include "../../include/aether/gb300/ag_tf64_trig.cuh"

typedef __float128 Q;
using namespace ag;
static bool differs(double a, double b) { return std::memcmp(&a, &b, 8) != 0 && !(a != a && b != b); }
static double ulps(double got, Q ref) {
    const double r = (double)ref;
    if (!differs(got, r)) return 0;
    if (got != got || std::isinf(got) || ref == 0) return std::numeric_limits<double>::infinity();
    int e;
    frexpq(fabsq(ref), &e);
    return (double)(fabsq((Q)got - ref) / ldexpq((Q)1, (e < -1021 ? -1021 : e) - 53));
}
static double exact_exp(double x) { return (double)expq((Q)x); }

int main() {
    const long N = 300000;
    std::mt19937_64 rng(23);
    std::uniform_real_distribution<double> u01(0.0, 1.0);
    auto sgn = [&] { return u01(rng) < 0.5 ? -1.0 : 1.0; };
    auto bits = [&](double lo, double hi) { return std::ldexp(1.0 + u01(rng), (int)std::floor(lo + (hi - lo) * u01(rng))); };
    const double special[] = {0.0, -0.0, 5e-324, -5e-324, 2.2e-308, 0x1p-1022, 0x1p-1021, 1.7976931348623157e308, 0x1p1023, 1.0, -1.0,
                              0x1p-41, 0x1p-40, 0x1p60, 0x1p61, 0x1.fffffffffffffp60, 0x1.fffffffffffffp-41, 709.78, 709.79, -708.39, -745.1,
                              -745.2, 710.0, -0.75, -0.9999999999999999, 88.0, -51.0, 1023.99, 1024.0, INFINITY, -INFINITY, NAN};
    const int S = sizeof special / sizeof *special;
    std::printf("{");
    auto line = [&](const char* name, long n, long differ, double worst) {
        std::printf("\"%s\": {\"n\": %ld, \"differ\": %ld, \"max_ulp\": %.6g, \"slow\": %ld}, ", name, n, differ, worst, g_slow);
        g_slow = 0;
    };
    // one argument: alone, and in either place of a pair
#define AG_EXACT(NAME, F, REF, DRAW, COUNT)                                                     \
    {                                                                                           \
        long d = 0;                                                                             \
        for (long i = 0; i < COUNT; ++i) {                                                      \
            const double x = DRAW, want = REF;                                                  \
            const double got = n64::F(x);                                                       \
            const long s = g_slow;                                                              \
            const e64::d2 p = n64::F(e64::d2{x, 2.0}), q = n64::F(e64::d2{2.0, x});             \
            g_slow = s;                                                                         \
            d += differs(got, want) || differs(p.a, want) || differs(q.b, want);                \
        }                                                                                       \
        line(NAME, COUNT, d, 0);                                                                \
    }
    AG_EXACT("sqrt", sqrt, std::sqrt(x), bits(-1022, 1024), N)
    AG_EXACT("rsqrt", rsqrt, 1.0 / std::sqrt(x), bits(-1022, 1024), N)
    AG_EXACT("sqrt_special", sqrt, std::sqrt(x), special[i], S)
    AG_EXACT("rsqrt_special", rsqrt, 1.0 / std::sqrt(x), special[i], S)
    AG_EXACT("sqrt_subnormal", sqrt, std::sqrt(x), std::ldexp(u01(rng), -1022), 2000)
    {
        long d = 0;
        for (long i = 0; i < N + S * S; ++i) {
            double a = sgn() * bits(-1022, 1024), b = sgn() * bits(-1022, 1024);
            if (i % 2) b = sgn() * a * bits(-60, 60);   // quotients that stay in range
            if (i >= N) a = special[(i - N) / S], b = special[(i - N) % S];
            if (i == N) line("div", N, d, 0), d = 0;
            const double want = a / b;
            d += differs(n64::div(a, b), want);
            const long s = g_slow;
            const e64::d2 p = n64::div(e64::d2{a, 1.0}, e64::d2{b, 3.0}), q = n64::div(e64::d2{1.0, a}, e64::d2{3.0, b});
            g_slow = s;
            d += differs(p.a, want) || differs(q.b, want);
        }
        line("div_special", S * S, d, 0);
    }
#define AG_ULP(NAME, F, DRAW, COUNT)                                                            \
    {                                                                                           \
        double worst = 0;                                                                       \
        for (long i = 0; i < COUNT; ++i) {                                                      \
            const double x = DRAW;                                                              \
            const Q want = F##q((Q)x);                                                          \
            const double got = n64::F(x);                                                       \
            const long s = g_slow;                                                              \
            const e64::d2 p = n64::F(e64::d2{x, 0.5}), q = n64::F(e64::d2{0.5, x});             \
            g_slow = s;                                                                         \
            for (double g : {got, p.a, q.b})                                                    \
                if (!(ulps(g, want) <= worst)) worst = ulps(g, want);                           \
        }                                                                                       \
        line(NAME, COUNT, 0, worst);                                                            \
    }
    AG_ULP("exp", exp, -708 + 1417 * u01(rng), N)
    AG_ULP("exp_tiny", exp, sgn() * bits(-1022, -38), N)
    AG_ULP("log", log, bits(-1022, 1024), N)
    AG_ULP("log1p", log1p, bits(50, 1024), N)
    AG_ULP("log1p_tiny", log1p, sgn() * bits(-1022, -38), N)
    AG_ULP("sin", sin, sgn() * bits(10, 22), N)
    AG_ULP("cos", cos, sgn() * bits(10, 22), N)
    AG_ULP("sin_multiples", sin, std::floor(2e6 * u01(rng) + 700) * 1.5707963267948966 * (1 + sgn() * bits(-53, -25)), N)
    AG_ULP("cos_multiples", cos, std::floor(2e6 * u01(rng) + 700) * 1.5707963267948966 * (1 + sgn() * bits(-53, -25)), N)
    AG_ULP("sin_huge", sin, sgn() * bits(21, 60), 20000)
    AG_ULP("cos_special", cos, special[i], S)
    AG_ULP("exp_special", exp, special[i], S)
    AG_ULP("log_special", log, special[i], S)
    AG_ULP("log1p_special", log1p, special[i], S)
    AG_ULP("exp_subnormal", exp, -745.2 + 37 * u01(rng), 2000)
    std::printf("\"end\": {\"n\": 1, \"differ\": 0, \"max_ulp\": 0, \"slow\": 0}}\n");
}
