// n64_ulp.cpp -- the errors of ag::n64's exp, log, log1p, sin, cos and normal
// draws against 113-bit arithmetic, per magnitude of the argument. A NaN or an
// infinity for a finite result counts as an infinite error and stays the
// worst. Prints one JSON object. Test infrastructure.
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
namespace ag {
inline double f_exp(double x) { return std::exp(x); }
inline double f_sin(double x) { return std::sin(x); }
inline double f_cos(double x) { return std::cos(x); }
namespace n64 {
inline double slow_sqrt(double x) { return std::sqrt(x); }
inline double slow_rsqrt(double x) { return 1.0 / std::sqrt(x); }
inline double slow_div(double a, double b) { return a / b; }
inline double slow_exp(double x) { return (double)expq((__float128)x); }
inline double slow_log(double x) { return (double)logq((__float128)x); }
inline double slow_log1p(double x) { return (double)log1pq((__float128)x); }
inline double slow_sin(double x) { return (double)sinq((__float128)x); }
inline double slow_cos(double x) { return (double)cosq((__float128)x); }
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
static double ulps(double got, Q ref) {
    if (got != got || std::isinf(got)) return std::numeric_limits<double>::infinity();
    if (ref == 0) return got == 0 ? 0.0 : std::numeric_limits<double>::infinity();
    int e;
    frexpq(fabsq(ref), &e);   // |ref| in [2^(e-1), 2^e): its ulp is 2^(e-53)
    return (double)(fabsq((Q)got - ref) / ldexpq((Q)1, (e < -1021 ? -1021 : e) - 53));
}

int main() {
    using namespace ag;
    const long N = 200000;
    std::mt19937_64 rng(17);
    std::uniform_real_distribution<double> u01(0.0, 1.0);
    auto logu = [&](double a, double b) { return std::exp2(a + (b - a) * u01(rng)); };
    auto sgn = [&] { return u01(rng) < 0.5 ? -1.0 : 1.0; };
    std::printf("{");
    auto sweep = [&](const char* name, auto draw, auto f, auto two, auto exact) {
        double worst = 0;
        for (long i = 0; i < N; ++i) {
            const double x = draw(), y = draw();
            const e64::d2 p = two(e64::d2{x, y});
            const Q ex = exact((Q)x), ey = exact((Q)y);
            for (double e : {ulps(f(x), ex), ulps(p.a, ex), ulps(p.b, ey)})
                if (!(e <= worst)) worst = e;   // never a NaN
        }
        std::printf("\"%s\": %.6g, ", name, worst);
    };
#define AG_SWEEP(NAME, F, DRAW) \
    sweep(NAME, [&] { return DRAW; }, [](double x) { return n64::F(x); }, [](e64::d2 x) { return n64::F(x); }, [](Q x) { return F##q(x); });
    AG_SWEEP("exp", exp, -55 + 145 * u01(rng))
    AG_SWEEP("exp_wide", exp, -700 + 1400 * u01(rng))
    AG_SWEEP("exp_small", exp, sgn() * logu(-60, 0))
    AG_SWEEP("log", log, logu(-45, 65))
    AG_SWEEP("log_wide", log, logu(-1000, 1000))
    AG_SWEEP("log_near_1", log, 1.0 + sgn() * logu(-52, -1))
    AG_SWEEP("log1p", log1p, logu(-45, 65))
    AG_SWEEP("log1p_wide", log1p, logu(-1000, 1000))
    AG_SWEEP("log1p_neg", log1p, -u01(rng))
    AG_SWEEP("log1p_neg_small", log1p, -logu(-60, 0))
    AG_SWEEP("sin", sin, sgn() * 1100 * u01(rng))
    AG_SWEEP("sin_wide", sin, sgn() * logu(9, 40))
    AG_SWEEP("sin_unit", sin, sgn() * 4 * u01(rng))
    AG_SWEEP("sin_small", sin, sgn() * logu(-60, 0))
    AG_SWEEP("sin_multiples", sin, std::floor(650 * u01(rng)) * 1.5707963267948966 * (1 + sgn() * logu(-53, -10)))
    AG_SWEEP("cos", cos, sgn() * 1100 * u01(rng))
    AG_SWEEP("cos_wide", cos, sgn() * logu(9, 40))
    AG_SWEEP("cos_unit", cos, sgn() * 4 * u01(rng))
    AG_SWEEP("cos_small", cos, sgn() * logu(-60, 0))
    AG_SWEEP("cos_multiples", cos, std::floor(650 * u01(rng)) * 1.5707963267948966 * (1 + sgn() * logu(-53, -10)))
    double worst = 0;
    for (long i = 0; i < N; ++i) {
        const double z = n64::normal(0x9E3779B97F4A7C15ull, (ag_u32)i, 3), s = n64::slow_normal(0x9E3779B97F4A7C15ull, (ag_u32)i, 3);
        const double e = z != z || s != s ? std::numeric_limits<double>::infinity() : std::fabs(z - s) / (1 + std::fabs(s)) * 0x1p53;
        if (!(e <= worst)) worst = e;
    }
    std::printf("\"normal\": %.6g}\n", worst);
}
