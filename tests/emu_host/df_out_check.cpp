// df_out_check.cpp -- host check of the reassembly of a double-float into a
// double (e64::out_double and out_bounded of ag_emu64.cuh) against the FP64 sum of the two
// floats (e64::to_double), for heads of every exponent and at powers of two,
// zeros and NaN. Prints one JSON object: per exponent of the head the results
// that differ, alone and as either sample of a pair, and those left to the native
// lane. Test infrastructure.
#include "host_shim.h"

#include <cstdio>
#include <random>

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
}  // namespace ag
#define AG_N64_HOST_CHECK
#include "../../include/aether/gb300/ag_emu64.cuh"

using namespace ag;

int main() {
    std::mt19937_64 rng(3);
    std::uniform_real_distribution<double> u01(0.0, 1.0);
    auto sgn = [&] { return u01(rng) < 0.5 ? -1.0 : 1.0; };
    auto differs = [](double a, double b) { return std::memcmp(&a, &b, 8) != 0 && !(a != a && b != b); };
    const e64::df one = e64::mk(1.5f, -0x1p-26f);
    long native = 0;   // values left to the native lane
    auto check = [&](e64::df v) {
        const double want = e64::to_double(v);
        bool ok = true;
        e64::b2 po = {true, true}, qo = {true, true};
        const double a = e64::out_bounded(v, ok);
        const e64::d2 p = e64::out_bounded(e64::pair(v, one), po), q = e64::out_bounded(e64::pair(one, v), qo);
        native += !ok;
        if (po.a != ok || qo.b != ok || !po.b || !qo.a) return true;
        return ok && (differs(a, want) || differs(p.a, want) || differs(q.b, want));
    };
    std::printf("{");
    for (int e = -126; e <= 126; ++e) {
        long d = 0, n = 0;
        for (int i = 0; i < 400; ++i) {
            const float m = i % 4 == 0 ? 1.0f : i % 4 == 1 ? 1.0f + 0x1p-23f : i % 4 == 2 ? 2.0f - 0x1p-23f : (float)(1.0 + 0.99 * u01(rng));
            const float hi = (float)(sgn() * std::exp2(e)) * m;
            // rests up to half a unit of the head, and one unit for a pair left unnormalised
            const float lo = (float)(hi * sgn() * std::exp2(i % 5 ? -25 - 24 * u01(rng) : -23.01));
            d += check(e64::mk(hi, i % 7 ? lo : 0.0f));
            ++n;
        }
        std::printf("\"%d\": {\"n\": %ld, \"differ\": %ld, \"native\": %ld}, ", e, n, d, native);
        native = 0;
    }
    long d = 0;
    for (float z : {0.0f, -0.0f})
        for (float w : {0.0f, -0.0f}) d += check(e64::mk(z, w));
    const float nan = __int_as_float(0x7fc00000);
    d += check(e64::mk(nan, nan)) + check(e64::mk(nan, 0.0f));
    std::printf("\"special\": {\"n\": 6, \"differ\": %ld, \"native\": %ld}}\n", d, native);
}
