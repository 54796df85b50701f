// ag_tf64_trig.cuh -- FP64-grade sine and cosine in triple-float arithmetic.
//
// Included by generated FP64-grade kernels (math = 3) with trigonometric
// nodes. x = q pi/2 + r with pi/2 in four parts (the first with 14 significant
// bits, so q P0 is exact for |q| < 2^10; about 87 bits in all); r = j/2048 + t
// with |t| <= 2^-12 and S_j, C_j = sin, cos(j/2048) from a table of three
// floats each; then, by quadrant, sin r = S (1 + cm1) + C st and
// cos r = C (1 + cm1) - S st with st = sin t = t (1 + c), c = -t^2/6 + t^4/120,
// and cm1 = cos t - 1 = -t^2/2 + t^4/24 (both corrections at most 2^-25, so
// double-float carries them to 2^-72).
//
// The reduction keeps every term exact: x.x - q P0 (Sterbenz), q P1 and q P2
// as two-products, and the terms of each level summed by two-sums, so r is
// good to about 2^-77 absolute. Lanes with |x| >= 2^10, or with |r| < 2^-22
// for q != 0 (x within 2^-22 of a nonzero multiple of pi/2, where 2^-77 would
// exceed 2^-55 of r), clear the range flag and are computed natively.
#pragma once

#include "ag_tf64.cuh"
#include "ag_tf64_trig_tables.cuh"

namespace ag {
namespace t64 {

// r = x - q pi/2, |r| <= pi/4 (a little beyond is fine).
__device__ __forceinline__ tf reduce_pio2(tf x, int& q, bool& ok) {
    const float qx = __fmul_rn(x.x, AG_TF_2OPI);
    const float qf = e64::rint_f(qx);
    q = e64::rint_i(qx);
    ok = ok && fabsf(x.x) < 1024.0f;
    const float a0 = __fmaf_rn(-qf, AG_TF_PIO2_0, x.x);   // exact: q P0 has <= 24 bits, Sterbenz
    const df p1 = two_prod(qf, AG_TF_PIO2_1);
    const df p2 = two_prod(qf, AG_TF_PIO2_2);
    const float p3 = __fmul_rn(qf, AG_TF_PIO2_3);
    // first level: a0 - q P1
    const df s = two_sum(a0, -p1.hi);
    // second level: s.lo, x.y, -p1.lo, -p2.hi, each summed exactly
    const df u = two_sum(x.y, -p1.lo);
    const df v = two_sum(s.lo, -p2.hi);
    const df w = two_sum(u.hi, v.hi);
    // third level: the errors of the second and the smallest terms, again by
    // two-sums; only the last roundings (2^-24 of 2^-62) are plain
    const df a = two_sum(u.lo, v.lo);
    const df b = two_sum(w.lo, x.z);
    const df c = two_sum(a.hi, b.hi);
    const float tail = __fadd_rn(__fadd_rn(__fadd_rn(a.lo, b.lo), c.lo), -__fadd_rn(p2.lo, p3));
    const df z = two_sum(c.hi, tail);
    // r = s.hi + w.hi + z.hi + z.lo, normalised (the parts can cancel)
    const df m = two_sum(w.hi, z.hi);
    const df n = two_sum(s.hi, m.hi);
    const df k = two_sum(n.lo, m.lo);
    const tf r = mk3(n.hi, k.hi, __fadd_rn(k.lo, z.lo));
    ok = ok && (q == 0 || fabsf(r.x) >= 2.384185791e-7f);   // 2^-22
    return renorm(r);
}

// One output of sin/cos at x = q pi/2 + r: by quadrant it is +-sin r or
// +-cos r, and both are A (1 + cm1) + B st with (A, B) = (S, C) for sin r and
// (C, -S) for cos r, so only the wanted one is evaluated.
__device__ __forceinline__ tf trig_(tf x, bool want_cos, bool& ok) {
    int q;
    const tf r = reduce_pio2(x, q, ok);
    const float jf = e64::rint_f(__fmul_rn(r.x, 2048.0f));
    int j = e64::rint_i(__fmul_rn(r.x, 2048.0f));
    j = j < -1664 ? -1664 : (j > 1664 ? 1664 : j);
    // t = r - j/2048: the leading difference is exact (Sterbenz, or j = 0)
    const tf t = renorm(mk3(__fmaf_rn(-jf, 4.8828125e-4f, r.x), r.y, r.z));
    const e64::f4 s0 = e64::ld4(kSinCos3, 2 * (j + AG_TF_SC_TAB_OFF));
    const e64::f4 s1 = e64::ld4(kSinCos3, 2 * (j + AG_TF_SC_TAB_OFF) + 1);
    const tf S = mk3(s0.x, s0.y, s0.z), C = mk3(s0.w, s1.x, s1.y);
    // st = t (1 + c), cm1 = -t^2/2 + t^4/24, both corrections in double-float
    const df tt = mk(t.x, t.y);
    const df t2 = e64::sqr(tt);
    const float t4 = __fmul_rn(t2.hi, t2.hi);
    const df c = e64::add_quick(e64::mul(t2, mk(-AG_TF_SIXTH_HI, -AG_TF_SIXTH_LO)), __fmul_rn(t4, 8.33333333e-3f));
    const df cm1 = e64::add_quick(e64::scale(t2, -0.5f), __fmul_rn(t4, 4.16666667e-2f));
    const df tc = e64::mul(tt, c);
    // st = t + t c: |t c| <= 2^-26 |t|
    const df h = fast_two_sum(t.x, tc.hi);
    const df g = two_sum(h.lo, t.y);
    const tf st = mk3(h.hi, g.hi, __fadd_rn(__fadd_rn(g.lo, t.z), tc.lo));
    const int quad = (q + (want_cos ? 1 : 0)) & 3;   // 0: sin r, 1: cos r, 2: -sin r, 3: -cos r
    const bool use_cos = quad & 1;
    const tf A = use_cos ? C : S;
    const tf B = use_cos ? neg(S) : C;
    // A leads: |A| >= sin(1/2048) > |B st| unless A = 0 (j = 0 for sin r);
    // A cm1 is 2^-25 of A at most
    const df Acm = e64::mul(mk(A.x, A.y), cm1);
    const tf v = add_lead(add_lead(A, mul(B, st)), mk3(Acm.hi, Acm.lo, 0.0f));
    return quad & 2 ? neg(v) : v;
}
__device__ __forceinline__ tf sin_(tf x, bool& ok) { return trig_(x, false, ok); }
__device__ __forceinline__ tf cos_(tf x, bool& ok) { return trig_(x, true, ok); }

}  // namespace t64

#if defined(__CUDACC__) || defined(__CUDACC_RTC__) || defined(AG_N64_HOST_CHECK)
namespace n64 {
#if defined(__CUDACC__) || defined(__CUDACC_RTC__)
__device__ AG_N64_NOINLINE double slow_sin(double x) { return ::sin(x); }
__device__ AG_N64_NOINLINE double slow_cos(double x) { return ::cos(x); }
__device__ AG_N64_NOINLINE double slow_normal(ag_u64 seed, ag_u32 g, ag_u32 c) { return ag::normal_f64(seed, g, c); }
#endif
// Below 2^-27, sin x = x and cos x = 1 to a quarter of an ulp.
__device__ __forceinline__ double sin(double x) {
    bool ok = true;
    const tf a = t64::from_double_ck(x, ok);
    const double r = join(t64::sin_(a, ok));
    if (((unsigned)__double2hiint(x) & 0x7fffffffu) < (996u << 20)) return x;
    return ok ? r : slow_sin(x);
}
__device__ __forceinline__ double cos(double x) {
    bool ok = true;
    const tf a = t64::from_double_ck(x, ok);
    const double r = join(t64::cos_(a, ok));
    if (((unsigned)__double2hiint(x) & 0x7fffffffu) < (996u << 20)) return 1.0;
    return ok ? r : slow_cos(x);
}

// The Box-Muller draw of ag::normal_f64 step by step: u and v are the
// reference's doubles, built in integers; log u, sqrt(-2 log u) and sin(pi v)
// are each rounded to a double as there, and two FP64 products are left of
// about 120 FP64 operations.
__device__ __forceinline__ double normal(ag_u64 seed, ag_u32 g, ag_u32 c) {
    const ag::q4 x = ag::philox_block(seed, g, c);
    // u = z 2^-53 + 2^-54 rounded to a double = w 2^-54, w < 2^54: exact below
    // 1/2, to even above it. Split in 24 + 23 + 7 bits from the leading one.
    const ag_u64 z = (ag_u64)x.x ^ ((ag_u64)x.y << 21);
    const ag_u64 w = z < (1ull << 52) ? 2ull * z + 1ull : 2ull * (z + (z & 1ull));
    const ag_u32 wh = (ag_u32)(w >> 32), wl = (ag_u32)w;
    const int lz = __clz((int)wh) - 10;   // -1 where u is 1
    bool ok = wh != 0u && lz >= 0;
    const ag_u32 nh = __funnelshift_l(wl, wh, (unsigned)lz), nl = wl << (lz & 31);
    const ag_u32 top = __funnelshift_l(nl, nh, 2u);   // bits 53..30
    const float my = __fsub_rn(__int_as_float((int)(0x4B000000u | ((nl >> 7) & 0x7fffffu))), 8388608.0f);
    const float mz = __fsub_rn(__int_as_float((int)(0x4B000000u | (nl & 127u))), 8388608.0f);
    const tf u = t64::mk3(__int_as_float((int)(((ag_u32)(126 - lz) << 23) | (top & 0x7fffffu))),
                          __fmul_rn(my, __int_as_float((int)((ag_u32)(80 - lz) << 23))),
                          __fmul_rn(mz, __int_as_float((int)((ag_u32)(73 - lz) << 23))));
    const double l = join(t64::log_s<false, t64::LOG_S0>(0.0f, u));   // < 0
    const double m2l = __hiloint2double((int)(((unsigned)__double2hiint(l) & 0x7fffffffu) + (1u << 20)), __double2loint(l));
    const double s = join(t64::sqrt_pos_(t64::from_double_ck(m2l, ok)));
    // v = zy 2^-52 + 2^-53 rounded = V 2^-53, V <= 2^54, its leading bit moved to bit 54
    const ag_u64 zy = (ag_u64)x.z ^ ((ag_u64)x.w << 21);
    const ag_u64 V = zy < (1ull << 52) ? 2ull * zy + 1ull : 2ull * (zy + (zy & 1ull));
    const ag_u32 vh = (ag_u32)(V >> 32), vl = (ag_u32)V;
    const int lv = __clz((int)vh) - 9;
    ok = ok && vh != 0u;
    const ag_u32 mh = __funnelshift_l(vl, vh, (unsigned)lv), ml = vl << (lv & 31);
    const double v = __hiloint2double((int)(((ag_u32)(1024 - lv) << 20) | ((mh >> 2) & 0xfffffu)),
                                      (int)((mh << 30) | (ml >> 2)));
    const tf p = t64::from_double_ck(__dmul_rn(v, 3.1415926535897932), ok);
    const double sv = join(t64::sin_(p, ok));
    const double r = __dmul_rn(s, sv);
    return ok ? r : slow_normal(seed, g, c);
}
}  // namespace n64

namespace t64 {
// N(0, 1) leaves of FP64-grade plans: the reference's formula, as in the
// native lowering, bit for bit.
template <bool U = false>
__device__ __forceinline__ tf normal_df(ag_u64 seed, ag_u32 g, ag_u32 c) {
    return dfc(n64::normal(seed, g, c));
}
}  // namespace t64
#endif

#ifdef AG_NATIVE_TF
__device__ __forceinline__ double f_sin(double x) { return n64::sin(x); }
__device__ __forceinline__ double f_cos(double x) { return n64::cos(x); }
__device__ __forceinline__ double drawn(double*, ag_u64 seed, ag_u32 g, ag_u32 c) { return n64::normal(seed, g, c); }
#endif
}  // namespace ag
