// tf_out_check.cpp -- host check of the reassembly of a triple-float into a
// double (t64::out_double of ag_tf64.cuh) where the value came out of a sum
// that cancelled, of a tie or of a value at the edge of its range. Prints one
// JSON object: per corpus the results that differ from the FP64 sum of the
// three floats (t64::to_double), the largest error against that exact sum in
// ulps of the result, and how many a generated kernel would hand to its native
// lane. Test infrastructure.
#include "host_shim.h"

#include <quadmath.h>

#include <cstdio>
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
inline double slow_exp(double x) { return std::exp(x); }
inline double slow_log(double x) { return std::log(x); }
inline double slow_log1p(double x) { return std::log1p(x); }
}  // namespace n64
}  // namespace ag
#define AG_N64_HOST_CHECK
#include "../../include/aether/gb300/ag_tf64.cuh"

typedef __float128 Q;
using namespace ag;
using t64::tf;

struct Stat {
    long n = 0, differ = 0, native = 0;
    double worst = 0;
    // `v` alone and as either sample of a pair with `w`
    void add(tf v, tf w) {
        ++n;
        if (!t64::out_ok(v)) {
            ++native;
            return;
        }
        const double want = t64::to_double(v);
        bool ok = true;
        e64::b2 po = {true, true}, qo = {true, true};
        const double one = t64::out_double(v, ok);
        const e64::d2 p = t64::out_double(t64::pair(v, w), po), q = t64::out_double(t64::pair(w, v), qo);
        if (!ok) {
            ++native;
            differ += po.a || qo.b;
            return;
        }
        differ += !(po.a && qo.b);
        const double got[3] = {one, p.a, q.b};
        const Q exact = (Q)v.x + (Q)v.y + (Q)v.z;
        bool d = false;
        for (double g : got) {
            d = d || !(g == want);
            int e;
            frexpq(fabsq(exact), &e);
            double u = exact == 0 ? (g == 0 ? 0.0 : 1e300) : (double)(fabsq((Q)g - exact) / ldexpq((Q)1, e - 53));
            if (u != u) u = 1e300;
            if (u > worst) worst = u;
        }
        differ += d;
    }
};
static bool first = true;
static void line(const char* name, int k, const Stat& s) {
    std::printf("%s\"%s_%d\": {\"n\": %ld, \"differ\": %ld, \"max_ulp\": %.6f, \"native\": %ld}", first ? "{" : ", ", name, k,
                s.n, s.differ, s.worst, s.native);
    first = false;
}
static tf split(double x) {
    bool ok = true;
    return t64::from_double_ck(x, ok);
}

int main() {
    std::mt19937_64 rng(5);
    std::uniform_real_distribution<double> u01(0.0, 1.0);
    auto logu = [&](double a, double b) { return std::exp2(a + (b - a) * u01(rng)); };
    auto sgn = [&] { return u01(rng) < 0.5 ? -1.0 : 1.0; };
    const long N = 20000;
    tf last = split(1.5);
    // v as the generated code hands it over: sums go through renorm first
    auto sum = [&](Stat& s, tf v) {
        const tf r = t64::renorm(v);
        s.add(r, last);
        last = r;
    };
    for (int k = 2; k <= 52; k += 2) {
        Stat diff, prod, logs;
        for (long i = 0; i < N; ++i) {
            const double a = sgn() * logu(-30, 50), b = a * (1.0 + sgn() * (0.5 + 1.5 * u01(rng)) * std::exp2(-k));
            sum(diff, t64::sub(split(a), split(b)));
            const double p = sgn() * logu(-10, 20), q = sgn() * logu(-10, 20), r = p * (1.0 + sgn() * logu(-k, 1 - k));
            const double t = p * q / r * (1.0 + sgn() * logu(-k, 1 - k));
            sum(prod, t64::sub(t64::mul(split(p), split(q)), t64::mul(split(r), split(t))));
            const double x = logu(-30, 50), y = x * (1.0 + (0.5 + u01(rng)) * std::exp2(-k));
            sum(logs, t64::sub(t64::log_(split(x)), t64::log_(split(y))));
        }
        line("difference", k, diff);
        line("products", k, prod);
        line("logarithms", k, logs);
    }
    Stat ties, whole, heads, edge;
    for (long i = 0; i < 10 * N; ++i) {
        // doubles of neighbouring exponents: every other sum is a tie
        const double a = sgn() * logu(-3, 3), b = sgn() * logu(-3, 3);
        sum(ties, t64::add(split(a), split(b)));
        sum(ties, t64::add(split(a), split(b * 0x1p-20)));
        // whole numbers, their heads' half units included
        const double m = std::floor(logu(0, 53)), m2 = std::floor(logu(0, 40));
        sum(whole, split(m));
        sum(whole, t64::sub(split(m + 1.0), split(m2)));
        // heads next to a power of two, rests of either sign up to half a unit
        const float x = (float)(sgn() * std::exp2(std::floor(150 * u01(rng)) - 70)) * (1.0f + (float)(i % 3 - 1) * 0x1p-23f);
        const float y = (float)(x * sgn() * logu(-40, -24.01)), z = (float)(y * sgn() * logu(-30, -23));
        heads.add(t64::mk3(x, i % 7 ? y : 0.0f, i % 5 ? z : 0.0f), last);
        // the lowest exponents that are not handed to the native lane, and the highest
        const int e = i % 2 ? -80 + int(i / 2 % 12) : 126 - int(i / 2 % 4);
        const float h = (float)(sgn() * std::exp2(e)) * (i % 3 ? 1.0f : (float)(1.0 + 0.99 * u01(rng)));
        edge.add(t64::mk3(h, (float)(h * sgn() * logu(-40, -24.01)), 0.0f), last);
    }
    // single operations as the generator hands them over: with their tail
    // renormalised after an exponential or a logarithm, as they are elsewhere
    Stat op[12], near;
    for (long i = 0; i < 5 * N; ++i) {
        const tf a = split(logu(-20, 20)), b = split(sgn() * logu(-20, 20)), c = split(logu(-2, 2)), d = split(logu(-2, 2));
        bool ok = true;
        const tf e = t64::exp_(split(sgn() * logu(-30, 5.5)), ok), l = t64::log_(split(logu(-30, 30))),
                 p = t64::log1p_(split(logu(-30, 30)));
        const tf v[12] = {t64::mul(a, b), t64::div(b, a), t64::recip(a), t64::sqrt_(a), t64::rsqrt_(a),
                          t64::sqrt_(t64::add_fast(t64::sqr(c), t64::sqr(d))), t64::add_fast(c, d), a,
                          t64::tail(e), t64::tail(l), t64::tail(p), t64::tail(t64::mul(e, l))};
        for (int k = 0; k < 12; ++k) op[k].add(v[k], last);
        near.add(t64::tail(t64::log_(split(1.0 + sgn() * logu(-50, -3)))), last);
    }
    line("near", 0, near);
    for (int k = 0; k < 12; ++k) line("op", k, op[k]);
    line("ties", 0, ties);
    line("whole", 0, whole);
    line("heads", 0, heads);
    line("edge", 0, edge);
    std::printf("}\n");
}
