// n64_check.cpp -- host check of the double functions of ag::n64
// (ag_tf64.cuh, ag_tf64_trig.cuh) against __float128 arithmetic. Prints one
// JSON object: per function the largest error in ulps of the exact result over
// a seeded corpus, and how many arguments took the out-of-line function. sqrt,
// rsqrt and div are compared with the correctly rounded host operations and
// report the number that differ. Test infrastructure.
#include "host_shim.h"

#include <quadmath.h>

#include <cstdio>
#include <random>

inline double __dmul_rn(double a, double b) { return a * b; }
inline int __float2int_rn(float f) { return (int)std::nearbyintf(f); }
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
// the reference's formula, each step rounded from its exact value
inline double slow_normal(ag_u64 seed, ag_u32 g, ag_u32 c) {
    ++g_slow;
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
    const double r = (double)ref;
    if (got == r || (got != got && r != r)) {
        if (got != got || std::isinf(got) || r == 0) return 0;
    }
    int e;
    frexpq(fabsq(ref), &e);   // |ref| in [2^(e-1), 2^e): its ulp is 2^(e-53)
    return (double)(fabsq((Q)got - ref) / ldexpq((Q)1, e - 53));
}

static bool first = true;
static void line(const char* name, long n, double worst, long differ) {
    std::printf("%s\"%s\": {\"n\": %ld, \"max_ulp\": %.6f, \"differ\": %ld, \"slow\": %ld}", first ? "{" : ", ", name, n,
                worst, differ, g_slow);
    first = false;
    g_slow = 0;
}

int main(int argc, char** argv) {
    const long N = argc > 1 ? std::atol(argv[1]) : 200000;
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> u01(0.0, 1.0);
    auto logu = [&](double a, double b) { return std::exp2(a + (b - a) * u01(rng)); };
    auto sgn = [&] { return u01(rng) < 0.5 ? -1.0 : 1.0; };
    auto sweep = [&](const char* name, auto draw, auto f, auto exact) {
        double worst = 0;
        for (long i = 0; i < N; ++i) {
            const double x = draw();
            const double e = ulps(f(x), exact((Q)x));
            if (!(e <= worst)) worst = e;
        }
        line(name, N, worst, 0);
    };
    auto count = [&](const char* name, auto draw, auto f, auto ref) {
        long d = 0;
        for (long i = 0; i < N; ++i) {
            const double x = draw();
            const double a = f(x), b = ref(x);
            d += !(a == b || (a != a && b != b));
        }
        line(name, N, 0, d);
    };
    using namespace ag;
    // near a power of two from either side, where the result's unit changes
    auto edge = [&] { return std::exp2(std::floor(40 * u01(rng) - 20)) * (1.0 + sgn() * logu(-53, -20)); };
    count("sqrt", [&] { return logu(-45, 65); }, [](double x) { return n64::sqrt(x); }, [](double x) { return std::sqrt(x); });
    count("sqrt_edge", edge, [](double x) { return n64::sqrt(x); }, [](double x) { return std::sqrt(x); });
    count("sqrt_square", [&] { const double y = std::floor(logu(0, 26)); return y * y; },
          [](double x) { return n64::sqrt(x); }, [](double x) { return std::sqrt(x); });
    count("rsqrt", [&] { return logu(-45, 65); }, [](double x) { return n64::rsqrt(x); },
          [](double x) { return 1.0 / std::sqrt(x); });
    count("rsqrt_edge", edge, [](double x) { return n64::rsqrt(x); }, [](double x) { return 1.0 / std::sqrt(x); });
    count("div", [&] { return sgn() * logu(-45, 65); }, [&](double x) { return n64::div(x, 3.0 - x); },
          [](double x) { return x / (3.0 - x); });
    count("div_edge", edge, [&](double x) { return n64::div(x * 1.5, x); }, [](double x) { return x * 1.5 / x; });
    {
        long d = 0;
        std::mt19937_64 r2(11);
        for (long i = 0; i < N; ++i) {
            const double a = sgn() * logu(-45, 65), b = sgn() * logu(-45, 65);
            d += n64::div(a, b) != a / b;
        }
        line("div_pairs", N, 0, d);
    }
    sweep("exp", [&] { return -55 + 145 * u01(rng); }, [](double x) { return n64::exp(x); }, [](Q x) { return expq(x); });
    sweep("exp_small", [&] { return sgn() * logu(-45, 0); }, [](double x) { return n64::exp(x); }, [](Q x) { return expq(x); });
    sweep("log", [&] { return logu(-45, 65); }, [](double x) { return n64::log(x); }, [](Q x) { return logq(x); });
    sweep("log_near_1", [&] { return 1.0 + sgn() * logu(-52, -1); }, [](double x) { return n64::log(x); },
          [](Q x) { return logq(x); });
    sweep("log1p", [&] { return logu(-45, 65); }, [](double x) { return n64::log1p(x); }, [](Q x) { return log1pq(x); });
    sweep("log1p_neg", [&] { return -u01(rng); }, [](double x) { return n64::log1p(x); }, [](Q x) { return log1pq(x); });
    sweep("log1p_neg_small", [&] { return -logu(-45, 0); }, [](double x) { return n64::log1p(x); }, [](Q x) { return log1pq(x); });
    for (int k = 0; k < 2; ++k) {
        auto f = [k](double x) { return k ? n64::cos(x) : n64::sin(x); };
        auto q = [k](Q x) { return k ? cosq(x) : sinq(x); };
        sweep(k ? "cos" : "sin", [&] { return sgn() * 1100 * u01(rng); }, f, q);
        sweep(k ? "cos_unit" : "sin_unit", [&] { return sgn() * 4 * u01(rng); }, f, q);
        sweep(k ? "cos_small" : "sin_small", [&] { return sgn() * logu(-60, 0); }, f, q);
        sweep(k ? "cos_multiples" : "sin_multiples",
              [&] { return std::floor(650 * u01(rng)) * 1.5707963267948966 * (1 + sgn() * logu(-53, -10)); }, f, q);
    }
    {   // the draw: log u, the root and the sine each rounded once, then their product
        double worst = 0;
        for (long i = 0; i < N; ++i) {
            const long before = g_slow;
            const double z = n64::normal(0x9E3779B97F4A7C15ull, (ag_u32)i, 3);
            const long s = g_slow;
            const double e = std::fabs(z - n64::slow_normal(0x9E3779B97F4A7C15ull, (ag_u32)i, 3)) / (1 + std::fabs(z)) * 0x1p53;
            g_slow = s;
            (void)before;
            if (!(e <= worst)) worst = e;
        }
        line("normal", N, worst, 0);
    }
    {   // the integer reassembly of a double-float against the sum in doubles,
        // unnormalised pairs and powers of two included; a pair of samples alike
        long d = 0;
        for (long i = 0; i < N; ++i) {
            float hi = (float)(sgn() * logu(-74, 120));
            if (i % 3 == 0) hi = (float)(sgn() * std::exp2(std::floor(190 * u01(rng) - 70)));
            float lo = (float)(hi * sgn() * logu(-60, -23));
            if (i % 5 == 0) lo = 0.0f;
            const e64::df v = e64::mk(hi, lo), w = e64::mk(-lo * 0.5f + hi, lo);
            const double want = (double)v.hi + (double)v.lo, want2 = (double)w.hi + (double)w.lo;
            d += e64::out_double(v) != want;
            const e64::d2 two = e64::out_double(e64::pair(v, w));
            d += two.a != want || two.b != want2;
        }
        line("reassemble", N, 0, d);
    }
    {   // two samples at a time give the same bits as one
        long d = 0;
        for (long i = 0; i < N; ++i) {
            const double x = sgn() * logu(-45, 65), y = sgn() * 4 * u01(rng);
            auto same = [](double a, double b) { return a == b || (a != a && b != b); };
#define AG_BOTH(F) { const e64::d2 r = n64::F(e64::d2{x, y}); d += !same(r.a, n64::F(x)) + !same(r.b, n64::F(y)); }
            AG_BOTH(sqrt) AG_BOTH(rsqrt) AG_BOTH(exp) AG_BOTH(log) AG_BOTH(log1p) AG_BOTH(sin) AG_BOTH(cos)
            const e64::d2 q = n64::div(e64::d2{x, y}, e64::d2{y, x});
            d += q.a != n64::div(x, y) || q.b != n64::div(y, x);
            const e64::d2 z = n64::normal(77, (ag_u32)i, (ag_u32)i + 1u, 2);
            d += z.a != n64::normal(77, (ag_u32)i, 2) || z.b != n64::normal(77, (ag_u32)i + 1u, 2);
        }
        line("pairs", N, 0, d);
    }
    std::printf("}\n");
}
