// ag_tf64_trig.cuh -- FP64-grade sine and cosine in triple-float arithmetic.
//
// Included by generated FP64-grade and native kernels with trigonometric nodes or
// normal draws. x = q pi/2 + r with pi/2 in four parts (the first with 14 significant
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

// |x| < 2^10, and |r| >= 2^-22 unless q = 0.
__device__ __forceinline__ void trig_range(float x, float r, int q, bool& ok) {
    ok = ok && fabsf(x) < 1024.0f && (q == 0 || fabsf(r) >= 2.384185791e-7f);
}
__device__ __forceinline__ void trig_range(f2 x, f2 r, i2 q, b2& ok) {
    trig_range(ln0(x), ln0(r), q.a, ok.a);
    trig_range(ln1(x), ln1(r), q.b, ok.b);
}
// r = x - q pi/2, |r| <= pi/4 (a little beyond is fine).
template <class F>
__device__ __forceinline__ tfT<F> reduce_pio2(tfT<F> x, typename lanes<F>::whole& q, typename lanes<F>::flag& ok) {
    const F qx = fmul(x.x, bc<F>(AG_TF_2OPI));
    const F qf = e64::rint_f(qx);
    q = e64::rint_i(qx);
    const F a0 = ffma(fneg(qf), bc<F>(AG_TF_PIO2_0), x.x);   // exact: q P0 has <= 24 bits, Sterbenz
    const dfT<F> p1 = two_prod(qf, bc<F>(AG_TF_PIO2_1));
    const dfT<F> p2 = two_prod(qf, bc<F>(AG_TF_PIO2_2));
    const F p3 = fmul(qf, bc<F>(AG_TF_PIO2_3));
    // first level: a0 - q P1
    const dfT<F> s = two_sum(a0, fneg(p1.hi));
    // second level: s.lo, x.y, -p1.lo, -p2.hi, each summed exactly
    const dfT<F> u = two_sum(x.y, fneg(p1.lo));
    const dfT<F> v = two_sum(s.lo, fneg(p2.hi));
    const dfT<F> w = two_sum(u.hi, v.hi);
    // third level: the errors of the second and the smallest terms, again by
    // two-sums; only the last roundings (2^-24 of 2^-62) are plain
    const dfT<F> a = two_sum(u.lo, v.lo);
    const dfT<F> b = two_sum(w.lo, x.z);
    const dfT<F> c = two_sum(a.hi, b.hi);
    const F tail = fsub(fadd(fadd(a.lo, b.lo), c.lo), fadd(p2.lo, p3));
    const dfT<F> z = two_sum(c.hi, tail);
    // r = s.hi + w.hi + z.hi + z.lo, normalised (the parts can cancel)
    const dfT<F> m = two_sum(w.hi, z.hi);
    const dfT<F> n = two_sum(s.hi, m.hi);
    const dfT<F> k = two_sum(n.lo, m.lo);
    const tfT<F> r = mk3(n.hi, k.hi, fadd(k.lo, z.lo));
    trig_range(x.x, r.x, q, ok);
    return renorm(r);
}

// r = x - q pi/2 for 2^10 <= |x| < 2^22, pi/2 as four floats, each the nearest
// to what the ones before it leave (103 bits). x.x - q C0 is exact (Sterbenz)
// but for q C0's rounding error, and its sum with x's other floats has at most
// 53 bits, two floats; q C1 and q C2 join as exact pairs. The sums' third floats
// round at 2^-73 in all, 2^-59 of |r| >= 2^-14; nearer arguments are flagged.
__device__ __forceinline__ tf reduce_wide(tf x, int& q, bool& ok) {
    const float qh = __fmul_rn(x.x, AG_TF_2OPI);
    const float ql = __fmaf_rn(x.y, AG_TF_2OPI, __fmaf_rn(x.x, 2.5682553e-08f, __fmaf_rn(x.x, AG_TF_2OPI, -qh)));
    const float q0 = e64::rint_f(qh);
    const float qf = __fadd_rn(q0, e64::rint_f(__fadd_rn(__fsub_rn(qh, q0), ql)));
    q = e64::rint_i(qf);
    const df p0 = two_prod(qf, 1.57079637f), p1 = two_prod(qf, -4.37113883e-08f), p2 = two_prod(qf, -1.71512451e-15f);
    const df s = two_sum(x.y, x.z), w = two_sum(__fsub_rn(x.x, p0.hi), s.hi);
    tf r = mk3(w.hi, __fadd_rn(w.lo, s.lo), 0.0f);
    r = add(r, mk3(-p0.lo, 0.0f, 0.0f));
    r = add(r, mk3(-p1.hi, -p1.lo, 0.0f));
    r = add(r, mk3(-p2.hi, -__fmaf_rn(qf, 1.0562999e-23f, p2.lo), 0.0f));
    r = renorm(r);
    ok = ok && fabsf(r.x) >= 6.103515625e-5f;
    return r;
}

// The table row of j/2048 at quadrant q: the pair (A, B) and the sign of the
// wanted output. By quadrant it is +-sin r or +-cos r, and both are
// A (1 + cm1) + B st with (A, B) = (S, C) for sin r and (C, -S) for cos r, so
// only the wanted one is evaluated.
template <class F>
struct trig_rows {
    tfT<F> A, B;
    typename lanes<F>::flag minus;
};
__device__ __forceinline__ trig_rows<float> trig_table(int j, int q, bool want_cos) {
    j = j < -1664 ? -1664 : (j > 1664 ? 1664 : j);
    const e64::f4 s0 = e64::ld4(kSinCos3, 2 * (j + AG_TF_SC_TAB_OFF));
    const e64::f4 s1 = e64::ld4(kSinCos3, 2 * (j + AG_TF_SC_TAB_OFF) + 1);
    const tf S = mk3(s0.x, s0.y, s0.z), C = mk3(s0.w, s1.x, s1.y);
    const int quad = (q + (want_cos ? 1 : 0)) & 3;   // 0: sin r, 1: cos r, 2: -sin r, 3: -cos r
    const bool use_cos = quad & 1;
    return trig_rows<float>{use_cos ? C : S, use_cos ? neg(S) : C, (quad & 2) != 0};
}
__device__ __forceinline__ trig_rows<f2> trig_table(i2 j, i2 q, bool want_cos) {
    const trig_rows<float> r = trig_table(j.a, q.a, want_cos), s = trig_table(j.b, q.b, want_cos);
    return trig_rows<f2>{pair(r.A, s.A), pair(r.B, s.B), b2{r.minus, s.minus}};
}
__device__ __forceinline__ tf neg_if(bool c, tf v) { return c ? neg(v) : v; }
__device__ __forceinline__ tf2 neg_if(b2 c, tf2 v) { return pair(neg_if(c.a, ln0(v)), neg_if(c.b, ln1(v))); }

// One output of sin/cos at x = q pi/2 + r.
template <class F>
__device__ __forceinline__ tfT<F> trig_reduced(tfT<F> r, typename lanes<F>::whole q, bool want_cos) {
    const F jx = fmul(r.x, bc<F>(2048.0f));
    const F jf = e64::rint_f(jx);
    // t = r - j/2048: the leading difference is exact (Sterbenz, or j = 0)
    const tfT<F> t = renorm(mk3(ffma(fneg(jf), bc<F>(4.8828125e-4f), r.x), r.y, r.z));
    const trig_rows<F> R = t64::trig_table(e64::rint_i(jx), q, want_cos);
    // st = t (1 + c), cm1 = -t^2/2 + t^4/24, both corrections in double-float
    const dfT<F> tt = mk(t.x, t.y);
    const dfT<F> t2 = e64::sqr(tt);
    const F t4 = fmul(t2.hi, t2.hi);
    const dfT<F> c = e64::add_quick(e64::mul(t2, mk(bc<F>(-AG_TF_SIXTH_HI), bc<F>(-AG_TF_SIXTH_LO))),
                                    fmul(t4, bc<F>(8.33333333e-3f)));
    const dfT<F> cm1 = e64::add_quick(e64::scale(t2, bc<F>(-0.5f)), fmul(t4, bc<F>(4.16666667e-2f)));
    const dfT<F> tc = e64::mul(tt, c);
    // st = t + t c: |t c| <= 2^-26 |t|
    const dfT<F> h = fast_two_sum(t.x, tc.hi);
    const dfT<F> g = two_sum(h.lo, t.y);
    const tfT<F> st = mk3(h.hi, g.hi, fadd(fadd(g.lo, t.z), tc.lo));
    // A leads: |A| >= sin(1/2048) > |B st| unless A = 0 (j = 0 for sin r);
    // A cm1 is 2^-25 of A at most
    const dfT<F> Acm = e64::mul(mk(R.A.x, R.A.y), cm1);
    const tfT<F> v = add_lead(add_lead(R.A, mul(R.B, st)), mk3(Acm.hi, Acm.lo, bc<F>(0.0f)));
    return neg_if(R.minus, v);
}
template <class F>
__device__ __forceinline__ tfT<F> trig_(tfT<F> x, bool want_cos, typename lanes<F>::flag& ok) {
    typename lanes<F>::whole q;
    const tfT<F> r = reduce_pio2(x, q, ok);
    return trig_reduced(r, q, want_cos);
}
template <class F>
__device__ __forceinline__ tfT<F> sin_(tfT<F> x, typename lanes<F>::flag& ok) {
    return trig_(x, false, ok);
}
template <class F>
__device__ __forceinline__ tfT<F> cos_(tfT<F> x, typename lanes<F>::flag& ok) {
    return trig_(x, true, ok);
}

}  // namespace t64

#if defined(__CUDACC__) || defined(__CUDACC_RTC__) || defined(AG_N64_HOST_CHECK)
namespace n64 {
#if defined(__CUDACC__) || defined(__CUDACC_RTC__)
__device__ __forceinline__ double slow_sin(double x) { return ::sin(x); }
__device__ __forceinline__ double slow_cos(double x) { return ::cos(x); }
__device__ AG_N64_NOINLINE double slow_normal(ag_u64 seed, ag_u32 g, ag_u32 c) { return ag::normal_f64(seed, g, c); }
#endif
template <class F>
__device__ __forceinline__ auto sin_core(tfT<F> a, typename lanes<F>::flag& ok) {
    return join(t64::sin_(a, ok));
}
template <class F>
__device__ __forceinline__ auto cos_core(tfT<F> a, typename lanes<F>::flag& ok) {
    return join(t64::cos_(a, ok));
}
// Arguments that sin_core and cos_core flag, out of line.
#define AG_N64_WIDE_TRIG(NAME, COS)                                        \
    __device__ AG_N64_NOINLINE double wide_##NAME(double x) {              \
        bool ok = exponent(x) - 1033u < 12u;   /* |x| in [2^10, 2^22) */   \
        if (!ok) return slow_##NAME(x);                                    \
        int q;                                                             \
        const tf r = t64::reduce_wide(split(x, ok), q, ok);                \
        const double v = join(t64::trig_reduced(r, q, COS));               \
        return ok ? v : slow_##NAME(x);                                    \
    }
AG_N64_WIDE_TRIG(sin, false)
AG_N64_WIDE_TRIG(cos, true)
// Below 2^-27, sin x = x and cos x = 1 to a quarter of an ulp.
__device__ __forceinline__ bool tiny(double x) {
    return ((unsigned)__double2hiint(x) & 0x7fffffffu) < (996u << 20);
}
#define AG_N64_TRIG(NAME, SMALL)                                           \
    __device__ __forceinline__ double NAME(double x) {                     \
        bool ok = true;                                                    \
        const tf a = split(x, ok);                                         \
        const double r = NAME##_core(a, ok);                               \
        return tiny(x) ? (SMALL) : ok ? r : wide_##NAME(x);                \
    }                                                                      \
    __device__ __forceinline__ double NAME##_rest(double x) {              \
        return tiny(x) ? (SMALL) : wide_##NAME(x);                         \
    }                                                                      \
    __device__ __forceinline__ d2 NAME(d2 x) {                             \
        b2 ok{true, true};                                                 \
        const t64::tf2 a = split(x, ok);                                   \
        d2 r = NAME##_core(a, ok);                                         \
        ok.a = ok.a && !tiny(x.a);                                         \
        ok.b = ok.b && !tiny(x.b);                                         \
        if (!(ok.a && ok.b)) {                                             \
            if (!ok.a) r.a = NAME##_rest(x.a);                             \
            if (!ok.b) r.b = NAME##_rest(x.b);                             \
        }                                                                  \
        return r;                                                          \
    }
AG_N64_TRIG(sin, x)
AG_N64_TRIG(cos, 1.0)

// The Box-Muller draw of ag::normal_f64 step by step: u and v are the
// reference's doubles, built in integers; log u, sqrt(-2 log u) and sin(pi v)
// are each rounded to a double as there, and two FP64 products are left of
// about 120 FP64 operations.
struct draw_words {
    tf u;
    double v;
};
__device__ __forceinline__ draw_words draw(ag_u64 seed, ag_u32 g, ag_u32 c, bool& ok) {
    const ag::q4 x = ag::philox_block(seed, g, c);
    draw_words d;
    // u = z 2^-53 + 2^-54 rounded to a double = w 2^-54, w < 2^54: exact below
    // 1/2, to even above it. Split in 24 + 23 + 7 bits from the leading one.
    const ag_u64 z = (ag_u64)x.x ^ ((ag_u64)x.y << 21);
    const ag_u64 w = z < (1ull << 52) ? 2ull * z + 1ull : 2ull * (z + (z & 1ull));
    const ag_u32 wh = (ag_u32)(w >> 32), wl = (ag_u32)w;
    const int lz = __clz((int)wh) - 10;   // -1 where u is 1
    const ag_u32 nh = __funnelshift_l(wl, wh, (unsigned)lz), nl = wl << (lz & 31);
    const ag_u32 top = __funnelshift_l(nl, nh, 2u);   // bits 53..30
    const float my = __fsub_rn(__int_as_float((int)(0x4B000000u | ((nl >> 7) & 0x7fffffu))), 8388608.0f);
    const float mz = __fsub_rn(__int_as_float((int)(0x4B000000u | (nl & 127u))), 8388608.0f);
    d.u = t64::mk3(__int_as_float((int)(((ag_u32)(126 - lz) << 23) | (top & 0x7fffffu))),
                   __fmul_rn(my, __int_as_float((int)((ag_u32)(80 - lz) << 23))),
                   __fmul_rn(mz, __int_as_float((int)((ag_u32)(73 - lz) << 23))));
    // v = zy 2^-52 + 2^-53 rounded = V 2^-53, V <= 2^54, its leading bit moved to bit 54
    const ag_u64 zy = (ag_u64)x.z ^ ((ag_u64)x.w << 21);
    const ag_u64 V = zy < (1ull << 52) ? 2ull * zy + 1ull : 2ull * (zy + (zy & 1ull));
    const ag_u32 vh = (ag_u32)(V >> 32), vl = (ag_u32)V;
    const int lv = __clz((int)vh) - 9;
    ok = ok && wh != 0u && lz >= 0 && vh != 0u;
    const ag_u32 mh = __funnelshift_l(vl, vh, (unsigned)lv), ml = vl << (lv & 31);
    d.v = __hiloint2double((int)(((ag_u32)(1024 - lv) << 20) | ((mh >> 2) & 0xfffffu)), (int)((mh << 30) | (ml >> 2)));
    return d;
}
// -2 x for x < 0
__device__ __forceinline__ double minus_twice(double x) {
    return __hiloint2double((int)(((unsigned)__double2hiint(x) & 0x7fffffffu) + (1u << 20)), __double2loint(x));
}
__device__ __forceinline__ d2 minus_twice(d2 x) { return d2{minus_twice(x.a), minus_twice(x.b)}; }
__device__ __forceinline__ double times(double x, double y) { return __dmul_rn(x, y); }
__device__ __forceinline__ d2 times(d2 x, d2 y) { return d2{__dmul_rn(x.a, y.a), __dmul_rn(x.b, y.b)}; }
template <class F, class D>
__device__ __forceinline__ D normal_core(tfT<F> u, D pv, typename lanes<F>::flag& ok) {
    const D l = join(t64::log_s<false, t64::LOG_S0>(bc<F>(0.0f), u));   // < 0
    const D s = join(t64::sqrt_pos_(split(minus_twice(l), ok)));
    return times(s, join(t64::sin_(split(pv, ok), ok)));
}
__device__ __forceinline__ double normal(ag_u64 seed, ag_u32 g, ag_u32 c) {
    bool ok = true;
    const draw_words d = draw(seed, g, c, ok);
    const double r = normal_core(d.u, __dmul_rn(d.v, 3.1415926535897932), ok);
    return ok ? r : slow_normal(seed, g, c);
}
__device__ __forceinline__ d2 normal(ag_u64 seed, ag_u32 g, ag_u32 h, ag_u32 c) {
    b2 ok{true, true};
    const draw_words d = draw(seed, g, c, ok.a), e = draw(seed, h, c, ok.b);
    d2 r = normal_core(t64::pair(d.u, e.u), d2{__dmul_rn(d.v, 3.1415926535897932), __dmul_rn(e.v, 3.1415926535897932)}, ok);
    if (!(ok.a && ok.b)) {
        if (!ok.a) r.a = slow_normal(seed, g, c);
        if (!ok.b) r.b = slow_normal(seed, h, c);
    }
    return r;
}
}  // namespace n64

namespace t64 {
// N(0, 1) leaves of FP64-grade plans: the reference's formula, as in the
// native lowering, bit for bit.
template <bool U = false>
__device__ __forceinline__ tf normal_df(ag_u64 seed, ag_u32 g, ag_u32 c) {
    return dfc(n64::normal(seed, g, c));
}
template <bool U = false>
__device__ __forceinline__ tf2 normal_df(ag_u64 seed, ag_u32 g, ag_u32 h, ag_u32 c) {
    const e64::d2 z = n64::normal(seed, g, h, c);
    return pair(dfc(z.a), dfc(z.b));
}
}  // namespace t64
#endif

#ifdef AG_NATIVE_TF
AG_N64_USE(sin)
AG_N64_USE(cos)
__device__ __forceinline__ double drawn(double*, ag_u64 seed, ag_u32 g, ag_u32 c) { return n64::normal(seed, g, c); }
__device__ __forceinline__ d2 drawn(double*, ag_u64 seed, ag_u32 g, ag_u32 h, ag_u32 c) {
    return n64::normal(seed, g, h, c);
}
#endif
}  // namespace ag
