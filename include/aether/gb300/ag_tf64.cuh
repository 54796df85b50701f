// ag_tf64.cuh -- FP64-grade expression math on the FP32 and integer pipes.
//
// Included by generated kernels lowered with math = 3, and by native ones (math =
// 0, and the native lanes of the others) that divide, take a root, exp, log, sine
// or cosine, or draw a normal (ag::n64 below). The double-float
// lowering (ag_emu64.cuh, math = 1) carries about 48 significant bits, tens
// of double ulps short of the FP64 contract; the native pipe meets the
// contract at a few per cent of HBM bandwidth. Here every double is split
// exactly into three floats (24 + 23 + 6 significant bits, integer operations
// only), the expression is evaluated in triple-float arithmetic (about 72
// bits, of which the operations keep well over 60), and each output is
// reassembled into a double in integers (out_double), one rounding of a value
// already exact to far below half an ulp.
//
// Representation: v = x + y + z with |y| of the order of ulp(x) and |z| of
// the order of 2^-24 |y|. The first two levels are combined by error-free
// transformations (two-sum, Fast2Sum, FMA two-product); the third is
// accumulated with plain float operations, whose roundings (2^-24 of a term
// of 2^-47 of the value) stay near 2^-71. The components are not kept
// strictly non-overlapping: every operation below accepts a y up to a few
// ulps of x and a z up to a few ulps of y. A sum that cancels leaves z large
// beside x, with the absolute error of its operands' scale; the generator
// renormalises such a value before it is reassembled.
//
// Range: inputs with magnitudes in [2^-40, 2^60] (and products the generator
// cannot prove to stay above 2^-80) keep every component a normal float;
// other lanes, non-finite or out-of-range outputs, and the functions without
// a triple-float kernel (tan, the inverse trigonometric and hyperbolic
// functions, pow and the rest) are computed with native FP64, so range and
// special values keep FP64 semantics.
//
// Methods (published; own code): Knuth two-sum, Dekker Fast2Sum, FMA
// two-product; Newton-Raphson square root, reciprocal square root and
// reciprocal, each a double-float result from ag_emu64.cuh refined by one
// step whose residual is formed exactly enough in triple-float; the
// table-driven logarithm of Tang (1990) with the reduction points of the
// double-float kernel and a third float on every table value; the
// table-driven exponential of Tang (1989); sine and cosine (ag_tf64_trig.cuh)
// by a four-part Cody-Waite reduction by pi/2 and a table of sin and cos at
// j/2048 (tables by gen_tf64_tables.py).
#pragma once

#include "ag_emu64.cuh"
#include "ag_tf64_tables.cuh"

namespace ag {
namespace t64 {

using e64::b2;
using e64::bc;
using e64::df;
using e64::dfT;
using e64::f2;
using e64::fadd;
using e64::fast_two_sum;
using e64::ffma;
using e64::fmul;
using e64::fneg;
using e64::fsub;
using e64::i2;
using e64::lanes;
using e64::ln0;
using e64::ln1;
using e64::mk;
using e64::pk;
using e64::two_prod;
using e64::two_sum;

// One sample (F = float) or two (F = f2, ag_emu64.cuh).
template <class F>
struct tfT {
    F x, y, z;
};
typedef tfT<float> tf;
typedef tfT<f2> tf2;

template <class F>
__device__ __forceinline__ tfT<F> mk3(F x, F y, F z) {
    tfT<F> r;
    r.x = x;
    r.y = y;
    r.z = z;
    return r;
}
__device__ __forceinline__ tf2 pair(tf a, tf b) { return mk3(pk(a.x, b.x), pk(a.y, b.y), pk(a.z, b.z)); }
__device__ __forceinline__ tf ln0(tf2 v) { return mk3(ln0(v.x), ln0(v.y), ln0(v.z)); }
__device__ __forceinline__ tf ln1(tf2 v) { return mk3(ln1(v.x), ln1(v.y), ln1(v.z)); }
__device__ __forceinline__ tf2 both(tf v) { return pair(v, v); }   // a value all samples share
template <class F>
__device__ __forceinline__ tfT<F> from_df(dfT<F> v) { return mk3(v.hi, v.lo, bc<F>(0.0f)); }
template <class F>
__device__ __forceinline__ tfT<F> neg(tfT<F> a) { return mk3(fneg(a.x), fneg(a.y), fneg(a.z)); }
template <class F>
__device__ __forceinline__ tfT<F> scale(tfT<F> a, F p2) {
    return mk3(fmul(a.x, p2), fmul(a.y, p2), fmul(a.z, p2));
}

// ---------------------------------------------------------------------------
// Arithmetic.
// ---------------------------------------------------------------------------
// a + b, any signs. The sum of the leading floats and of the second floats
// are exact pairs; their errors and the third floats form the third level.
// Under cancellation the result keeps an absolute error near 2^-71 of the
// larger operand.
template <class F>
__device__ __forceinline__ tfT<F> add(tfT<F> a, tfT<F> b) {
    const dfT<F> s = two_sum(a.x, b.x);
    const dfT<F> t = two_sum(a.y, b.y);
    const dfT<F> u = two_sum(s.lo, t.hi);
    const F z = fadd(fadd(t.lo, u.lo), fadd(a.z, b.z));
    const dfT<F> w = two_sum(s.hi, u.hi);
    return mk3(w.hi, w.lo, z);
}
template <class F>
__device__ __forceinline__ tfT<F> sub(tfT<F> a, tfT<F> b) { return add(a, neg(b)); }
// a + b for operands of one sign: |s.hi| is at least either leading float,
// so the last combination is a Fast2Sum.
template <class F>
__device__ __forceinline__ tfT<F> add_fast(tfT<F> a, tfT<F> b) {
    const dfT<F> s = two_sum(a.x, b.x);
    const dfT<F> t = two_sum(a.y, b.y);
    const dfT<F> u = two_sum(s.lo, t.hi);
    const F z = fadd(fadd(t.lo, u.lo), fadd(a.z, b.z));
    const dfT<F> w = fast_two_sum(s.hi, u.hi);
    return mk3(w.hi, w.lo, z);
}
// a + b where a leads: |a.x| >= |b.x| (or a.x = 0) and |a + b| >= |a| / 2, so
// the leading floats join by Fast2Sum and the result cannot cancel.
template <class F>
__device__ __forceinline__ tfT<F> add_lead(tfT<F> a, tfT<F> b) {
    const dfT<F> s = fast_two_sum(a.x, b.x);
    const dfT<F> t = two_sum(a.y, b.y);
    const dfT<F> u = two_sum(s.lo, t.hi);
    const F z = fadd(fadd(t.lo, u.lo), fadd(a.z, b.z));
    const dfT<F> w = fast_two_sum(s.hi, u.hi);
    return mk3(w.hi, w.lo, z);
}
// A plan's root has no cheaper form here: its reassembly in integers wants the
// first two floats normalised.
template <class F>
__device__ __forceinline__ tfT<F> add_fast_u(tfT<F> a, tfT<F> b) { return add_fast(a, b); }

// a b: the three products of the first two levels as exact pairs, the
// third-level products by FMA; the dropped terms are below 2^-70 of the
// product.
template <class F>
__device__ __forceinline__ tfT<F> mul(tfT<F> a, tfT<F> b) {
    const dfT<F> p = two_prod(a.x, b.x);
    const dfT<F> q1 = two_prod(a.x, b.y);
    const dfT<F> q2 = two_prod(a.y, b.x);
    const F r = ffma(a.y, b.y, ffma(a.x, b.z, fmul(a.z, b.x)));
    const dfT<F> s = two_sum(q1.hi, q2.hi);
    const dfT<F> u = two_sum(p.lo, s.hi);
    const F z = fadd(fadd(fadd(q1.lo, q2.lo), fadd(s.lo, u.lo)), r);
    const dfT<F> w = fast_two_sum(p.hi, u.hi);   // |u.hi| is about 2^-23 |p.hi| at most
    return mk3(w.hi, w.lo, z);
}
template <class F>
__device__ __forceinline__ tfT<F> mul(tfT<F> a, F f) {
    const dfT<F> p = two_prod(a.x, f);
    const dfT<F> q = two_prod(a.y, f);
    const dfT<F> u = two_sum(p.lo, q.hi);
    const F z = ffma(a.z, f, fadd(q.lo, u.lo));
    const dfT<F> w = fast_two_sum(p.hi, u.hi);
    return mk3(w.hi, w.lo, z);
}
template <class F>
__device__ __forceinline__ tfT<F> sqr(tfT<F> a) {
    const dfT<F> p = two_prod(a.x, a.x);
    const F x2 = fadd(a.x, a.x);   // exact
    const dfT<F> q = two_prod(x2, a.y);
    const F r = ffma(a.y, a.y, fmul(x2, a.z));
    const dfT<F> u = two_sum(p.lo, q.hi);
    const F z = fadd(fadd(q.lo, u.lo), r);
    const dfT<F> w = fast_two_sum(p.hi, u.hi);
    return mk3(w.hi, w.lo, z);
}
// The square of a double-float as a triple-float (no third input float).
template <class F>
__device__ __forceinline__ tfT<F> sqr_df(dfT<F> a) {
    const dfT<F> p = two_prod(a.hi, a.hi);
    const dfT<F> q = two_prod(fadd(a.hi, a.hi), a.lo);
    const dfT<F> u = two_sum(p.lo, q.hi);
    const F z = ffma(a.lo, a.lo, fadd(q.lo, u.lo));
    const dfT<F> w = fast_two_sum(p.hi, u.hi);
    return mk3(w.hi, w.lo, z);
}
// Products read only by sums: every sum above takes any overlap, so the same
// value serves.
template <class F>
__device__ __forceinline__ tfT<F> sqr_u(tfT<F> a) { return sqr(a); }

// Products below 2^-80 in magnitude would push the third float toward the
// subnormal range; such lanes take the native path.
#define AG_TF_MIN 8.2718061255302767e-25f   // 2^-80
__device__ __forceinline__ tf ck(tf v, bool& ok) {
    ok = ok && fabsf(v.x) >= AG_TF_MIN;
    return v;
}
__device__ __forceinline__ tf2 ck(tf2 v, b2& ok) {
    ok.a = ok.a && fabsf(ln0(v.x)) >= AG_TF_MIN;
    ok.b = ok.b && fabsf(ln1(v.x)) >= AG_TF_MIN;
    return v;
}

// (x, y, z) with the overlap of y and z folded into y: y + z as an exact
// pair, then x with its leading part (two-sums, so x may be the smaller).
template <class F>
__device__ __forceinline__ tfT<F> renorm(tfT<F> v) {
    const dfT<F> s = two_sum(v.y, v.z);
    const dfT<F> w = two_sum(v.x, s.hi);
    return mk3(w.hi, w.lo, s.lo);
}
// The same for y and z alone, of a value whose x leads its y already.
template <class F>
__device__ __forceinline__ tfT<F> tail(tfT<F> v) {
    const dfT<F> s = two_sum(v.y, v.z);
    return mk3(v.x, s.hi, s.lo);
}

// Reciprocal: the double-float reciprocal (about 2^-47) refined by one Newton
// step r' = r + r e, e = 1 - y r. y r is within 2^-46 of 1, so 1 - x of the
// product is exact (Sterbenz) and its second and third floats join by
// subtractions that are exact or round at 2^-70.
template <class F>
__device__ __forceinline__ tfT<F> recip(tfT<F> y) {
    const dfT<F> r = e64::recip_t(mk(y.x, y.y));
    const tfT<F> m = mul(y, from_df(r));
    const F e = fsub(fsub(fsub(bc<F>(1.0f), m.x), m.y), m.z);
    return mk3(r.hi, r.lo, fmul(r.hi, e));
}
template <class F>
__device__ __forceinline__ tfT<F> div(tfT<F> a, tfT<F> b) { return mul(a, recip(b)); }

// Comparisons by the sign of the difference: the leading float of a sum
// carries its sign unless the whole sum is zero at the first two levels.
__device__ __forceinline__ int sgn_(tf d) {
    const float v = d.x != 0.0f ? d.x : (d.y != 0.0f ? d.y : d.z);
    return v > 0.0f ? 1 : (v < 0.0f ? -1 : 0);
}
__device__ __forceinline__ bool gt(tf a, tf b) { return sgn_(sub(a, b)) > 0; }
__device__ __forceinline__ bool lt(tf a, tf b) { return sgn_(sub(a, b)) < 0; }
__device__ __forceinline__ bool ge(tf a, tf b) { return sgn_(sub(a, b)) >= 0; }
__device__ __forceinline__ bool le(tf a, tf b) { return sgn_(sub(a, b)) <= 0; }
__device__ __forceinline__ bool eq(tf a, tf b) { return sgn_(sub(a, b)) == 0; }
__device__ __forceinline__ bool ne(tf a, tf b) { return sgn_(sub(a, b)) != 0; }
#define AG_T64_CMP2(NAME) \
    __device__ __forceinline__ b2 NAME(tf2 x, tf2 y) { return b2{NAME(ln0(x), ln0(y)), NAME(ln1(x), ln1(y))}; }
AG_T64_CMP2(gt)
AG_T64_CMP2(lt)
AG_T64_CMP2(ge)
AG_T64_CMP2(le)
AG_T64_CMP2(eq)
AG_T64_CMP2(ne)
#undef AG_T64_CMP2
__device__ __forceinline__ tf2 sel(b2 c, tf2 x, tf2 y) {
    return pair(c.a ? ln0(x) : ln0(y), c.b ? ln1(x) : ln1(y));
}

// ---------------------------------------------------------------------------
// double <-> triple-float.
// ---------------------------------------------------------------------------
// The exact split of a double with |x| in [2^-40, 2^60] (the flag is cleared
// outside): x takes the implicit bit and the top 23 stored bits (the same
// integer work as the double-float split), y the next 23 bits and z the last
// 6, each made a float by the 2^23 exponent trick (no conversion unit) and
// scaled by a power of two built from x's exponent field.
__device__ __forceinline__ tf from_double_ck(double v, bool& ok) {
    const unsigned h32 = (unsigned)__double2hiint(v);
    const unsigned l32 = (unsigned)__double2loint(v);
    const unsigned t = (h32 & 0x7fffffffu) - (896u << 20);
    ok = ok && t - (87u << 20) <= (101u << 20) - 1u;   // double exponent in [-40, 60]
    const unsigned hb = __funnelshift_l(l32, t, 3) | (h32 & 0x80000000u);
    const unsigned se = hb & 0xff800000u;   // sign and exponent field of x
    const float my = __fsub_rn(__int_as_float((int)(0x4B000000u | ((l32 >> 6) & 0x7fffffu))), 8388608.0f);
    const float mz = __fsub_rn(__int_as_float((int)(0x4B000000u | (l32 & 63u))), 8388608.0f);
    // bit k of the stored mantissa weighs 2^(e - 52 + k): y's lowest bit is
    // bit 6, z's bit 0
    const float y = __fmul_rn(my, __int_as_float((int)(se - (46u << 23))));
    const float z = __fmul_rn(mz, __int_as_float((int)(se - (52u << 23))));
    return mk3(__int_as_float((int)hb), y, z);
}
__device__ __forceinline__ tf2 from_double_ck(double v, double w, b2& ok) {
    return pair(from_double_ck(v, ok.a), from_double_ck(w, ok.b));
}
// Any double (runtime scalars, literals, native results): the split by
// conversions on the FP64 pipe, exact for normal values.
__device__ __forceinline__ tf dfc(double v) {
    const float x = __double2float_rn(v);
    if (!isfinite(x)) return mk3(x, 0.0f, 0.0f);
    const double r = v - (double)x;
    const float y = __double2float_rn(r);
    return mk3(x, y, __double2float_rn(r - (double)y));
}
// y + z in a double is exact whenever their exponents lie within 29 of each
// other, and otherwise off by at most 2^-53 of y (about 2^-77 of x): the
// result is x + y + z rounded once, to far below half an ulp.
__device__ __forceinline__ double to_double(tf v) {
    return __dadd_rn((double)v.x, __dadd_rn((double)v.y, (double)v.z));
}
__device__ __forceinline__ e64::d2 to_double(tf2 v) { return e64::d2{to_double(ln0(v)), to_double(ln1(v))}; }
__device__ __forceinline__ double as_d(tf v) { return to_double(v); }
// An output whose three floats were all normal: |x| in [2^-80, 2^127).
__device__ __forceinline__ bool out_ok(tf v) {
    const unsigned e = ((unsigned)__float_as_int(v.x) >> 23) & 0xffu;
    return e - 47u <= 206u;
}

// ---------------------------------------------------------------------------
// Square root and reciprocal square root.
// ---------------------------------------------------------------------------
// a > 0. s = the double-float root (about 2^-47), then s' = s + (a - s^2)
// y/2 with y ~ 1/sqrt(a) the float seed. The residual is about 2^-47 a and is
// needed to 2^-12 of itself: a.x - s.hi^2 is exact (Sterbenz), and the terms
// of the second level, each up to 2^-23 a and cancelling to the residual, are
// summed by two-sums.
template <class F>
__device__ __forceinline__ tfT<F> sqrt_pos_(tfT<F> a) {
    const F y = e64::rsqrt_seed(a.x);
    const F s0 = fmul(a.x, y);
    const dfT<F> p0 = two_prod(s0, s0);
    const F r0 = fadd(fsub(fsub(a.x, p0.hi), p0.lo), a.y);
    const F hy = fmul(bc<F>(0.5f), y);
    const dfT<F> s = fast_two_sum(s0, fmul(r0, hy));
    const dfT<F> P = two_prod(s.hi, s.hi);
    const dfT<F> Q = two_prod(fadd(s.hi, s.hi), s.lo);
    const dfT<F> e1 = two_sum(fsub(a.x, P.hi), a.y);
    const dfT<F> e2 = two_sum(e1.hi, fneg(P.lo));
    const dfT<F> e3 = two_sum(e2.hi, fneg(Q.hi));
    const F small = fsub(fadd(fadd(e1.lo, e2.lo), fadd(e3.lo, a.z)),
                                  ffma(s.lo, s.lo, Q.lo));
    const F R = fadd(e3.hi, small);
    return mk3(s.hi, s.lo, fmul(R, hy));
}
template <class F>
__device__ __forceinline__ tfT<F> sqrt_(tfT<F> a) {
    const tfT<F> r = sqrt_pos_(a);
    return mk3(e64::or_zero(a.x, r.x), e64::or_zero(a.x, r.y), e64::or_zero(a.x, r.z));
}
template <class F>
__device__ __forceinline__ tfT<F> sqrt_nn_(tfT<F> a) { return sqrt_(a); }
// a > 0. y = the double-float rsqrt (about 2^-47), then y' = y + y e / 2 with
// e = 1 - a y^2 formed like the reciprocal's residual.
template <class F>
__device__ __forceinline__ tfT<F> rsqrt_(tfT<F> a) {
    const dfT<F> y = e64::rsqrt_t(mk(a.x, a.y));
    const tfT<F> m = mul(a, sqr_df(y));
    const F e = fsub(fsub(fsub(bc<F>(1.0f), m.x), m.y), m.z);
    return mk3(y.hi, y.lo, fmul(fmul(y.hi, e), bc<F>(0.5f)));
}

// ---------------------------------------------------------------------------
// log and log1p: y = s + a = 2^e m, m in [0.75, 1.5), i = round(1024 (m - 1)),
// A = c_i 2^-e, t = s A - 1 + a A (|t| <= 2^-10.6), and
// log y = e ln2 - log c_i + log1p(t), log1p(t) = t + t^2 Q(t) with
// Q = -1/2 + t/3 - t^2/4 + t^3/5 - t^4/6 + t^5/7 (the next term is below
// 2^-66 of t). t^2 Q is about 2^-12 of t, so it is formed in double-float
// (2^-46 of itself, 2^-58 of t) with the coefficient 1/3 as a float pair.
// ---------------------------------------------------------------------------
struct log_row {
    float A;
    tf L, E;
    bool valid;
};
__device__ __forceinline__ log_row log_reduce(float yh) {
    const int bits = __float_as_int(yh);
    int e = ((bits >> 23) & 0xff) - 127;
    int mb = (bits & 0x007fffff) | 0x3f800000;
    if (bits & 0x00400000) {   // m >= 1.5: use m/2 and e+1
        mb -= 0x00800000;
        e += 1;
    }
    const float m = __int_as_float(mb);
    const int i = e64::rint_i(__fmaf_rn(m, 1024.0f, -1024.0f)) + AG_TF_LOG_TAB_OFF;
    const e64::f4 cl = e64::ld4(kLogCL3, i), ep = e64::ld4(kLn2Mul3, e + AG_TF_LN2_TAB_OFF);
    log_row r;
    r.A = __int_as_float((int)((unsigned)__float_as_int(cl.x) - ((unsigned)e << 23)));   // c 2^-e, exact
    r.L = mk3(cl.y, cl.z, cl.w);
    r.E = mk3(ep.x, ep.y, ep.z);
    r.valid = yh > 0.0f && e > -120 && e < 120;
    return r;
}
template <class F>
struct log_rows {
    F A;
    tfT<F> L, E;
    typename lanes<F>::flag valid;
};
__device__ __forceinline__ log_rows<float> log_tables(float yh) {
    const log_row r = log_reduce(yh);
    return log_rows<float>{r.A, r.L, r.E, r.valid};
}
__device__ __forceinline__ log_rows<f2> log_tables(f2 yh) {
    const log_row r = log_reduce(ln0(yh)), s = log_reduce(ln1(yh));
    return log_rows<f2>{pk(r.A, s.A), pair(r.L, s.L), pair(r.E, s.E), b2{r.valid, s.valid}};
}
__device__ __forceinline__ tf or_nan(bool ok, tf v) { return ok ? v : mk3(__int_as_float(0x7fc00000), 0.0f, 0.0f); }
__device__ __forceinline__ tf2 or_nan(b2 ok, tf2 v) { return pair(or_nan(ok.a, ln0(v)), or_nan(ok.b, ln1(v))); }

enum { LOG_S0 = 0, LOG_S1 = 1 };
template <bool checked, int MODE, class F>
__device__ __forceinline__ tfT<F> log_s(F s, tfT<F> a) {
    const log_rows<F> R = t64::log_tables(fadd(s, a.x));
    const tfT<F> aA = mul(a, R.A);
    tfT<F> t;
    if (MODE == LOG_S0) {
        // a A is within 2^-10 of 1: its leading float less 1 is exact
        const dfT<F> d = two_sum(fsub(aA.x, bc<F>(1.0f)), aA.y);
        t = mk3(d.hi, d.lo, aA.z);
    } else {
        const dfT<F> B = two_sum(R.A, bc<F>(-1.0f));   // A - 1 exactly
        t = add(mk3(B.hi, B.lo, bc<F>(0.0f)), aA);
    }
    // t's third float can be far above an ulp of its second when t is small
    // (a A within 2^-24 of 1 leaves a's third float beside a tiny leading
    // part), and the series below reads t's first two floats only
    t = renorm(t);
    // P = t^2 Q in double-float
    const F th = t.x;
    const dfT<F> tt = mk(t.x, t.y);
    const F r = ffma(th, ffma(th, ffma(th, bc<F>(0.142857143f), bc<F>(-0.166666667f)), bc<F>(0.2f)), bc<F>(-0.25f));
    const dfT<F> G = e64::add_quick(mk(bc<F>(AG_TF_THIRD_HI), bc<F>(AG_TF_THIRD_LO)), e64::mul(tt, r));
    const dfT<F> Q = e64::add_quick(mk(bc<F>(-0.5f), bc<F>(0.0f)), e64::mul(tt, G));
    const dfT<F> P = e64::mul(e64::sqr(tt), Q);
    // T = t + P: |P| < |t| / 2^11
    const dfT<F> h = fast_two_sum(t.x, P.hi);
    const dfT<F> k = two_sum(h.lo, t.y);
    const tfT<F> T = mk3(h.hi, k.hi, fadd(fadd(k.lo, t.z), P.lo));
    // e ln2 - log c_i, each from its table as three floats. |e ln2| >= ln2 >
    // 0.29 >= |log c_i| unless e = 0, and |-log c_i| >= 2^-10 >= 2 |T| unless
    // i = 0 (then the leading term is 0): both sums are led by their first term.
    const tfT<F> res = add_lead(add_lead(R.E, R.L), T);
    return checked ? or_nan(R.valid, res) : res;
}
template <class F>
__device__ __forceinline__ tfT<F> log_(tfT<F> a) {
    return log_s<true, LOG_S0>(bc<F>(0.0f), a);
}
template <class F>
__device__ __forceinline__ tfT<F> log1p_(tfT<F> a) {
    return log_s<true, LOG_S1>(bc<F>(1.0f), a);
}
// log1p of an argument known to be >= 0 and within the input range
template <class F>
__device__ __forceinline__ tfT<F> log1p_nn_(tfT<F> a) {
    return log_s<false, LOG_S1>(bc<F>(1.0f), a);
}

// ---------------------------------------------------------------------------
// Simple nodes, Philox draws and the bridge to native FP64.
// ---------------------------------------------------------------------------
__device__ __forceinline__ tf abs_(tf a) { return sgn_(a) < 0 ? neg(a) : a; }
__device__ __forceinline__ tf sign_(tf a) { return mk3((float)sgn_(a), 0.0f, 0.0f); }
__device__ __forceinline__ tf min_(tf a, tf b) { return lt(b, a) ? b : a; }
__device__ __forceinline__ tf max_(tf a, tf b) { return gt(b, a) ? b : a; }
__device__ __forceinline__ tf2 abs_(tf2 x) { return pair(abs_(ln0(x)), abs_(ln1(x))); }
__device__ __forceinline__ tf2 sign_(tf2 x) { return pair(sign_(ln0(x)), sign_(ln1(x))); }
__device__ __forceinline__ tf2 min_(tf2 x, tf2 y) { return pair(min_(ln0(x), ln0(y)), min_(ln1(x), ln1(y))); }
__device__ __forceinline__ tf2 max_(tf2 x, tf2 y) { return pair(max_(ln0(x), ln0(y)), max_(ln1(x), ln1(y))); }
// (2w + 1) 2^-33: exact in the first two floats.
__device__ __forceinline__ tf draw01_df(ag_u64 seed, ag_u32 g, ag_u32 c) {
    return from_df(e64::draw01_df(seed, g, c));
}
__device__ __forceinline__ tf2 draw01_df(ag_u64 seed, ag_u32 g, ag_u32 h, ag_u32 c) {
    return pair(draw01_df(seed, g, c), draw01_df(seed, h, c));
}
// ---------------------------------------------------------------------------
// exp: x = k ln2/64 + r, |r| <= ln2/128, e^x = 2^(k >> 6) T_(k & 63) (1 + p),
// T_j = 2^(j/64) from a table of three floats, p = e^r - 1 = r + r^2 Q(r),
// Q = 1/2 + r/6 + r^2/24 + r^3/120 + r^4/720 + r^5/5040 (the next term is
// below 2^-66). r = x - k (ln2/64) with ln2/64 as three floats (k < 2^13, so
// the product is good to 2^-63 absolute, the sum exact to 2^-64). r^2 Q is at
// most 2^-16: formed in double-float (2^-46 of itself), with 1/6 and 1/24 as
// float pairs where their products with r sit within 2^-12 of the terms
// before them. The flag is cleared outside -55 < x < 87, where 2^(k >> 6) or
// the result's third float would leave the normal floats (the native lane
// computes those).
// ---------------------------------------------------------------------------
__device__ __forceinline__ tf exp_table(int k) {
    const e64::f4 tv = e64::ld4(kExp2Tab3, k & 63);
    return mk3(tv.x, tv.y, tv.z);
}
__device__ __forceinline__ tf2 exp_table(i2 k) { return pair(exp_table(k.a), exp_table(k.b)); }
// e^x = 2^(k >> 6) exp_mantissa(x, k), the mantissa in [1, 2) but for rounding.
template <class F>
__device__ __forceinline__ tfT<F> exp_mantissa(tfT<F> x, typename lanes<F>::whole& k) {
    const F kx = fmul(x.x, bc<F>(AG_TF_INV_LN2_64));
    const F kf = e64::rint_f(kx);
    k = e64::rint_i(kx);
    const tfT<F> ln2 = mk3(bc<F>(AG_TF_LN2_64_X), bc<F>(AG_TF_LN2_64_Y), bc<F>(AG_TF_LN2_64_Z));
    const tfT<F> r = renorm(sub(x, mul(ln2, kf)));
    const dfT<F> rr = mk(r.x, r.y);
    const F rh = r.x;
    const F J = ffma(rh, ffma(rh, bc<F>(1.98412698e-4f), bc<F>(1.38888889e-3f)), bc<F>(8.33333333e-3f));
    const dfT<F> H = e64::add_quick(mk(bc<F>(AG_TF_24TH_HI), bc<F>(AG_TF_24TH_LO)), fmul(rh, J));
    const dfT<F> G = e64::add_quick(mk(bc<F>(AG_TF_SIXTH_HI), bc<F>(AG_TF_SIXTH_LO)), e64::mul(rr, H));
    const dfT<F> Q = e64::add_quick(mk(bc<F>(0.5f), bc<F>(0.0f)), e64::mul(rr, G));
    const dfT<F> P = e64::mul(e64::sqr(rr), Q);
    // p = r + P: |P| <= r^2 < |r|
    const dfT<F> h = fast_two_sum(r.x, P.hi);
    const dfT<F> m = two_sum(h.lo, r.y);
    const tfT<F> p = mk3(h.hi, m.hi, fadd(fadd(m.lo, r.z), P.lo));
    const tfT<F> T = t64::exp_table(k);
    // T >= 1 leads T p (|p| < 2^-7)
    return add_lead(T, mul(T, p));
}
template <class F>
__device__ __forceinline__ tfT<F> exp_(tfT<F> x, typename lanes<F>::flag& ok) {
    e64::within(x.x, -55.0f, 87.0f, ok);
    typename lanes<F>::whole k;
    const tfT<F> res = exp_mantissa(x, k);
    return scale(res, e64::p2f(e64::exp_power(k)));
}
#define AG_T64_NATIVE1(NAME)                                                                   \
    __device__ __forceinline__ tf nat_##NAME(tf x) { return dfc(ag::f_##NAME(as_d(x))); }      \
    __device__ __forceinline__ tf2 nat_##NAME(tf2 x) { return pair(nat_##NAME(ln0(x)), nat_##NAME(ln1(x))); }
#define AG_T64_NATIVE2(NAME)                                                                   \
    __device__ __forceinline__ tf nat_##NAME(tf a, tf b) { return dfc(ag::f_##NAME(as_d(a), as_d(b))); } \
    __device__ __forceinline__ tf2 nat_##NAME(tf2 x, tf2 y) {                                  \
        return pair(nat_##NAME(ln0(x), ln0(y)), nat_##NAME(ln1(x), ln1(y)));                   \
    }
AG_T64_NATIVE1(expm1)
AG_T64_NATIVE1(exp2)
AG_T64_NATIVE1(log2)
AG_T64_NATIVE1(log10)
AG_T64_NATIVE1(tan)
AG_T64_NATIVE1(asin)
AG_T64_NATIVE1(acos)
AG_T64_NATIVE1(atan)
AG_T64_NATIVE1(tanh)
AG_T64_NATIVE1(sinh)
AG_T64_NATIVE1(cosh)
AG_T64_NATIVE1(floor)
AG_T64_NATIVE1(ceil)
AG_T64_NATIVE1(trunc)
AG_T64_NATIVE1(cbrt)
AG_T64_NATIVE1(erf)
AG_T64_NATIVE2(pow)
AG_T64_NATIVE2(atan2)
AG_T64_NATIVE2(hypot)
#undef AG_T64_NATIVE1
#undef AG_T64_NATIVE2

}  // namespace t64
namespace y64 = t64;   // the spelling of a plan's two-sample code

#if defined(__CUDACC__) || defined(__CUDACC_RTC__) || defined(AG_N64_HOST_CHECK)
// ---------------------------------------------------------------------------
// double -> double functions of the native lowering (math = 0), evaluated in
// triple-float arithmetic and rounded once. The FP64 pipe issues two lanes a
// clock and SM against 110 of the FP32 pipe, so CUDA's FP64 functions (15 to
// 60 operations on it) bound every plan that calls one; these use none of it.
// sqrt, rsqrt and div are correctly rounded: a value closer to a rounding
// boundary than the evaluation's own error is handed to the FP64 pipe. log,
// log1p, exp, sin and cos are within 0.52 ulp, under CUDA's 1 to 2; sin and cos
// 0.76 beside multiples of pi/2 (0.63 seen in 9 10^6 arguments as near as the
// fast path takes). Arguments outside the triple-float range are scaled into it
// out of line (wide_* below); subnormals, overflow, infinities, NaN and sines
// beyond 2^22 take CUDA's function there. Measured: a + b c + sin(a) exp(-c c) over 2^20
// three-component samples, 232 us with CUDA's functions, 65 us with these; a
// fill of 3 uniform components and one N(0, 1) draw for 10^7 samples, 1555 and
// 267 us.
// ---------------------------------------------------------------------------
namespace n64 {
using t64::tf;

// Zeros answer at once: sparse data has many.
__device__ __forceinline__ bool is_zero(double x) {
    return (((unsigned)__double2hiint(x) & 0x7fffffffu) | (unsigned)__double2loint(x)) == 0u;
}
#if defined(__CUDACC__) || defined(__CUDACC_RTC__)
#define AG_N64_NOINLINE __noinline__
__device__ __forceinline__ double slow_sqrt(double x) { return __dsqrt_rn(x); }
__device__ __forceinline__ double slow_rsqrt(double x) { return __ddiv_rn(1.0, __dsqrt_rn(x)); }
__device__ __forceinline__ double slow_div(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ double slow_exp(double x) { return ::exp(x); }
__device__ __forceinline__ double slow_log(double x) { return ::log(x); }
__device__ __forceinline__ double slow_log1p(double x) { return ::log1p(x); }
__device__ __forceinline__ double fma_rn(double x, double y, double z) { return __fma_rn(x, y, z); }
#else
#define AG_N64_NOINLINE inline
inline double fma_rn(double x, double y, double z) { return std::fma(x, y, z); }
#endif

using e64::d2;
using e64::plus;
using t64::b2;
using t64::bc;
using t64::f2;
using t64::fadd;
using t64::fmul;
using t64::fsub;
using t64::i2;
using t64::lanes;
using t64::ln0;
using t64::ln1;
using t64::pk;
using t64::tfT;

// One double or a pair of them, and the triple-float type of as many.
__device__ __forceinline__ tf split(double v, bool& ok) { return t64::from_double_ck(v, ok); }
__device__ __forceinline__ t64::tf2 split(d2 v, b2& ok) { return t64::from_double_ck(v.a, v.b, ok); }

using e64::join_bits;
using e64::to_int;
// x + y + z rounded to a double in integers and floats alone: the double of x
// with (y + z) in its units added to its bits. Needs |x| in [2^-75, 2^100) and
// |y| within a few ulps of x. `g` is the last part of (y + z) before it is
// rounded to the integer `i`: |g - i| near 1/2 is a value near a boundary.
template <class F>
__device__ __forceinline__ auto join(tfT<F> v, F& g, typename lanes<F>::whole& i) {
    const F S = e64::join_scale(v.x, fadd(v.y, v.z));
    const F Y = fmul(v.y, S), Z = fmul(v.z, S);   // exact scalings
    const typename lanes<F>::whole i1 = to_int(Y);
    g = fadd(fsub(Y, e64::to_f(i1)), Z);
    i = to_int(g);
    return join_bits(v.x, plus(i1, i));
}
template <class F>
__device__ __forceinline__ auto join(tfT<F> v) {
    F g;
    typename lanes<F>::whole i;
    return join(v, g, i);
}
// The same, clearing `ok` within 2^-12 of an ulp of a rounding boundary (the
// triple-float sqrt and recip are good to 2^-15 of one, the quotient to 2^-14).
// One lane in 2048 then takes the function out of line. 2^-9 sent one in 256,
// some lane of every eighth warp, to 20 FP64 operations and more: the large
// streaming expression over 2^24 x 3 samples took 1180 us so, 945 now, 3x3
// inverses of 2^22 samples 282 and 237.
template <class F>
__device__ __forceinline__ auto join_exact(tfT<F> v, typename lanes<F>::flag& ok) {
    F g;
    typename lanes<F>::whole i;
    const auto r = join(v, g, i);
    e64::within(fsub(g, e64::to_f(i)), -0.499755859375f, 0.499755859375f, ok);
    return r;
}

template <class F>
__device__ __forceinline__ auto sqrt_core(tfT<F> a, typename lanes<F>::flag& ok) {
    e64::within(a.x, 0.0f, 3e38f, ok);
    return join_exact(t64::sqrt_pos_(a), ok);
}
// 1 / sqrt(x), each step rounded (the host spelling of math/root.h:64-76)
template <class F>
__device__ __forceinline__ auto rsqrt_core(tfT<F> a, typename lanes<F>::flag& ok) {
    const auto s = sqrt_core(a, ok);
    return join_exact(t64::recip(split(s, ok)), ok);
}
template <class F>
__device__ __forceinline__ auto div_core(tfT<F> x, tfT<F> y, typename lanes<F>::flag& ok) {
    const tfT<F> q = t64::mul(x, t64::recip(y));
    e64::within(e64::fabs_(q.x), 2.7105054e-20f, 7.9228163e28f, ok);   // |q| in (2^-65, 2^96)
    return join_exact(q, ok);
}
template <class F>
__device__ __forceinline__ auto exp_core(tfT<F> a, typename lanes<F>::flag& ok) {
    e64::within(a.x, -50.0f, 3e38f, ok);
    return join(t64::exp_(a, ok));
}
template <class F>
__device__ __forceinline__ auto log_core(tfT<F> a, typename lanes<F>::flag& ok) {
    const tfT<F> l = t64::log_s<false, t64::LOG_S0>(bc<F>(0.0f), a);
    e64::within(a.x, 0.0f, 3e38f, ok);
    e64::within(e64::fabs_(l.x), 0.0f, 3e38f, ok);   // log 1 = 0 has no leading float
    return join(l);
}
template <class F>
__device__ __forceinline__ auto log1p_core(tfT<F> a, typename lanes<F>::flag& ok) {
    e64::within(a.x, -0.75f, 3e38f, ok);   // nearer to -1 the reduced argument cancels
    return join(t64::log_s<false, t64::LOG_S1>(bc<F>(1.0f), a));
}
// Arguments the triple-float split does not take, out of line: the double is
// brought to an exponent near 0 in integers, the same evaluation runs on it, and
// the exponent goes back into the result's bits. What is left (values beside a
// rounding boundary, subnormals, overflow, negative or non-finite arguments) is
// CUDA's function's. sqrt of 3 x 2^22 doubles near 1e-20: 93 us, CUDA's
// 187, near 1 50; quotients 132, 183 and 66; exp of -200 to -60 190 and 370; logarithms
// near 1e25 184 and 705; sines up to 1e5 249 and 434 (ag_tf64_trig.cuh).
__device__ __forceinline__ unsigned exponent(double x) { return ((unsigned)__double2hiint(x) >> 20) & 0x7ffu; }
// exponent + k, mantissa and sign unchanged
__device__ __forceinline__ double times_2(double x, int k) {
    return __hiloint2double(__double2hiint(x) + (int)((unsigned)k << 20), __double2loint(x));
}
__device__ __forceinline__ bool normal_exponent(int e) { return (unsigned)(e - 1) < 2046u; }
__device__ __forceinline__ bool in_split(unsigned e) { return e - 983u <= 100u; }   // |x| in [2^-40, 2^61)
__device__ AG_N64_NOINLINE double wide_sqrt(double x) {
    if (is_zero(x)) return x;
    const unsigned e = (unsigned)__double2hiint(x) >> 20;   // the sign is its top bit
    if (in_split(e) || !normal_exponent((int)e)) return slow_sqrt(x);
    const int k = ((int)e - 1023) & ~1;
    bool ok = true;
    const tf a = split(times_2(x, -k), ok);
    const double r = sqrt_core(a, ok);
    return ok ? times_2(r, k / 2) : slow_sqrt(x);
}
__device__ AG_N64_NOINLINE double wide_rsqrt(double x) {
    const unsigned e = (unsigned)__double2hiint(x) >> 20;
    if (in_split(e) || !normal_exponent((int)e)) return slow_rsqrt(x);
    const int k = ((int)e - 1023) & ~1;
    bool ok = true;
    const tf a = split(times_2(x, -k), ok);
    const double r = rsqrt_core(a, ok);
    return ok ? times_2(r, -(k / 2)) : slow_rsqrt(x);
}
__device__ AG_N64_NOINLINE double wide_div(double x, double y) {
    const int ex = (int)exponent(x), ey = (int)exponent(y), k = ex - ey;
    if (is_zero(x) && normal_exponent(ey)) return __hiloint2double((__double2hiint(x) ^ __double2hiint(y)) & (int)0x80000000, 0);
    // both in the split's range and the quotient in div_core's: beside a boundary
    const bool near = in_split((unsigned)ex) && in_split((unsigned)ey) && k > -64 && k < 95;
    if (near || !normal_exponent(ex) || !normal_exponent(ey)) return slow_div(x, y);
    bool ok = true;
    const tf a = split(times_2(x, 1023 - ex), ok), b = split(times_2(y, 1023 - ey), ok);
    const double r = div_core(a, b, ok);
    return ok && normal_exponent((int)exponent(r) + k) ? times_2(r, k) : slow_div(x, y);
}
// Below 2^-40, e^x = 1 + x to 2^-81; elsewhere the power of two joins the bits.
__device__ AG_N64_NOINLINE double wide_exp(double x) {
    const unsigned e = exponent(x);
    if (e < 983u) return __dadd_rn(1.0, x);
    bool ok = e < 1033u;   // |x| < 2^10: the multiple of ln2/64 is exact
    const tf a = split(x, ok);
    int k;
    const double r = join(t64::exp_mantissa(a, k));
    return ok && normal_exponent((int)exponent(r) + (k >> 6)) ? times_2(r, k >> 6) : slow_exp(x);
}
// log x = k ln2 + log(x 2^-k); outside the split's range the first term leads.
__device__ AG_N64_NOINLINE double wide_log(double x) {
    const unsigned e = (unsigned)__double2hiint(x) >> 20;
    if (in_split(e) || !normal_exponent((int)e)) return slow_log(x);
    const int k = (int)e - 1023;
    bool ok = true;
    const tf a = split(times_2(x, -k), ok);
    const tf ln2 = t64::mk3(64.0f * AG_TF_LN2_64_X, 64.0f * AG_TF_LN2_64_Y, 64.0f * AG_TF_LN2_64_Z);
    return join(t64::add_lead(t64::mul(ln2, (float)k), t64::log_s<false, t64::LOG_S0>(0.0f, a)));
}
// Below 2^-40, log(1 + x) = x - x^2/2 to 2^-81 of it; above 2^60 it is log x to
// 2^-13 of an ulp; between -1 and -1/2, 1 + x is exact.
__device__ AG_N64_NOINLINE double wide_log1p(double x) {
    const unsigned e = exponent(x);
    if (is_zero(x)) return x;
    if (e < 983u) return fma_rn(__dmul_rn(x, -0.5), x, x);
    if (x > 0.0 && e < 2047u && !in_split(e)) return wide_log(x);
    if (x > -1.0 && x <= -0.5) {
        const double y = __dadd_rn(1.0, x);
        if (!in_split(exponent(y))) return wide_log(y);
        bool ok = true;
        const tf a = split(y, ok);
        const double r = log_core(a, ok);
        if (ok) return r;
    }
    return slow_log1p(x);
}
#define AG_N64_FUNCTION(NAME)                                              \
    __device__ __forceinline__ double NAME(double x) {                     \
        bool ok = true;                                                    \
        const tf a = split(x, ok);                                         \
        const double r = NAME##_core(a, ok);                               \
        return ok ? r : wide_##NAME(x);                                    \
    }                                                                      \
    __device__ __forceinline__ d2 NAME(d2 x) {                             \
        b2 ok{true, true};                                                 \
        const t64::tf2 a = split(x, ok);                                   \
        d2 r = NAME##_core(a, ok);                                         \
        if (!(ok.a && ok.b)) {                                             \
            if (!ok.a) r.a = wide_##NAME(x.a);                             \
            if (!ok.b) r.b = wide_##NAME(x.b);                             \
        }                                                                  \
        return r;                                                          \
    }
AG_N64_FUNCTION(sqrt)
AG_N64_FUNCTION(rsqrt)
AG_N64_FUNCTION(exp)
AG_N64_FUNCTION(log)
AG_N64_FUNCTION(log1p)
__device__ __forceinline__ double div(double x, double y) {
    bool ok = true;
    const tf a = split(x, ok), b = split(y, ok);
    const double r = div_core(a, b, ok);
    return ok ? r : wide_div(x, y);
}
__device__ __forceinline__ d2 div(d2 x, d2 y) {
    b2 ok{true, true};
    const t64::tf2 a = split(x, ok), b = split(y, ok);
    d2 r = div_core(a, b, ok);
    if (!(ok.a && ok.b)) {
        if (!ok.a) r.a = wide_div(x.a, y.a);
        if (!ok.b) r.b = wide_div(x.b, y.b);
    }
    return r;
}
}  // namespace n64

namespace t64 {
// Whether x + y + z can be put together in integers, given Y and Z, its lower
// parts in twice the unit of the double's last place: |x| in [2^-75, 2^127),
// |Y| <= 2^28 (the next float's distance: the sum stays in x's binade), and
// |Z| <= 2^8, so that a float holds what is rounded to 2^-15 of a unit. False
// for a NaN.
__device__ __forceinline__ bool join_fits(float x, float Y, float Z) {
    return e64::join_head<1>(x) && fabsf(Y) <= 268435456.0f && fabsf(Z) <= 256.0f;
}
__device__ __forceinline__ b2 join_fits(f2 x, f2 Y, f2 Z) {
    return b2{join_fits(ln0(x), ln0(Y), ln0(Z)), join_fits(ln1(x), ln1(Y), ln1(Z))};
}
// x + y + z rounded once to nearest even, without the FP64 pipe (five operations
// of it in to_double), where join_fits holds: where the parts overlap no more
// than a product or a root of normalised operands leaves them. The generator hands
// over a sum that may cancel renormalised (12 FP32 operations), and what comes from
// an exponential or a logarithm, whose third float is the rest of a double-float
// series, with its tail renormalised (6). Y is rounded to an even number of
// units and what is left by an addition to 1.5 2^22, whose last place is half of
// Y's unit, so that a tie goes to the even double.
__device__ __forceinline__ int half_units(float g) { return __float_as_int(__fadd_rn(g, 6291456.0f)) - 0x4AC00000; }
__device__ __forceinline__ i2 half_units(f2 g) {
    const f2 t = fadd(g, bc<f2>(6291456.0f));
    return i2{__float_as_int(ln0(t)) - 0x4AC00000, __float_as_int(ln1(t)) - 0x4AC00000};
}
template <class F>
__device__ __forceinline__ auto out_join(tfT<F> v, typename lanes<F>::flag& fits) {
    const F S = e64::join_scale<1>(v.x, fadd(v.y, v.z));
    const F Y = fmul(v.y, S), Z = fmul(v.z, S);   // exact scalings
    const typename lanes<F>::whole h = e64::to_int(Y);
    const F g = fadd(fsub(Y, e64::to_f(h)), Z);
    fits = join_fits(v.x, Y, Z);
    return e64::join_bits(v.x, e64::plus(e64::plus(h, h), half_units(g)));
}
// Where parts that seldom overlap did: the value with its tail renormalised.
__device__ __forceinline__ void take(bool& fits, double& r, bool f, double v) {
    if (!fits) r = v, fits = f;
}
__device__ __forceinline__ void take(b2& fits, e64::d2& r, b2 f, e64::d2 v) {
    take(fits.a, r.a, f.a, v.a);
    take(fits.b, r.b, f.b, v.b);
}
template <class F, class D>
__device__ AG_N64_NOINLINE void out_again(tfT<F> v, typename lanes<F>::flag& fits, D& r) {
    typename lanes<F>::flag f;
    const D w = out_join(tail(v), f);
    take(fits, r, f, w);
}
// A plan's output. `ok` is cleared where the parts do not fit; the lane runs
// natively there.
template <bool RETRY = false, class F>
__device__ __forceinline__ auto out_double(tfT<F> v, typename lanes<F>::flag& ok) {
    typename lanes<F>::flag fits;
    auto r = out_join(v, fits);
    if (RETRY && !e64::all_of(fits)) out_again(v, fits, r);
    ok = e64::both_of(ok, fits);
    return r;
}
// The same for a root whose bounds keep it in range: zero and NaN (the root of a
// negative number) leave as they are.
template <bool RETRY = false, class F>
__device__ __forceinline__ auto out_bounded(tfT<F> v, typename lanes<F>::flag& ok) {
    typename lanes<F>::flag fits;
    auto r = out_join(v, fits);
    if (!e64::all_of(fits)) {
        if (RETRY) out_again(v, fits, r);
        r = e64::or_zero_nan(v.x, r, fits, ok);
    }
    return r;
}
}  // namespace t64
#endif

#ifdef AG_NATIVE_TF
// The functions and operations of native plans, for one sample and for two.
using e64::b2;
using e64::both;
using e64::d2;
__device__ __forceinline__ d2 rn_add(d2 x, d2 y) { return d2{rn_add(x.a, y.a), rn_add(x.b, y.b)}; }
__device__ __forceinline__ d2 rn_sub(d2 x, d2 y) { return d2{rn_sub(x.a, y.a), rn_sub(x.b, y.b)}; }
__device__ __forceinline__ d2 rn_mul(d2 x, d2 y) { return d2{rn_mul(x.a, y.a), rn_mul(x.b, y.b)}; }
__device__ __forceinline__ double rn_fma(double x, double y, double z) { return __fma_rn(x, y, z); }
__device__ __forceinline__ d2 rn_fma(d2 x, d2 y, d2 z) { return d2{__fma_rn(x.a, y.a, z.a), __fma_rn(x.b, y.b, z.b)}; }
__device__ __forceinline__ double rn_neg(double x) { return -x; }
__device__ __forceinline__ d2 rn_neg(d2 x) { return d2{-x.a, -x.b}; }
__device__ __forceinline__ double ln0(d2 x) { return x.a; }
__device__ __forceinline__ double ln1(d2 x) { return x.b; }
__device__ __forceinline__ d2 sel(b2 c, d2 x, d2 y) { return d2{c.a ? x.a : y.a, c.b ? x.b : y.b}; }
__device__ __forceinline__ b2 gt(d2 x, d2 y) { return b2{x.a > y.a, x.b > y.b}; }
__device__ __forceinline__ b2 lt(d2 x, d2 y) { return b2{x.a < y.a, x.b < y.b}; }
__device__ __forceinline__ b2 ge(d2 x, d2 y) { return b2{x.a >= y.a, x.b >= y.b}; }
__device__ __forceinline__ b2 le(d2 x, d2 y) { return b2{x.a <= y.a, x.b <= y.b}; }
__device__ __forceinline__ b2 eq(d2 x, d2 y) { return b2{x.a == y.a, x.b == y.b}; }
__device__ __forceinline__ b2 ne(d2 x, d2 y) { return b2{x.a != y.a, x.b != y.b}; }
#define AG_D2_UNARY(NAME) \
    __device__ __forceinline__ d2 f2_##NAME(d2 x) { return d2{f_##NAME(x.a), f_##NAME(x.b)}; }
#define AG_D2_BINARY(NAME) \
    __device__ __forceinline__ d2 f2_##NAME(d2 x, d2 y) { return d2{f_##NAME(x.a, y.a), f_##NAME(x.b, y.b)}; }
AG_D2_UNARY(abs)
AG_D2_UNARY(sign)
AG_D2_UNARY(expm1)
AG_D2_UNARY(exp2)
AG_D2_UNARY(log2)
AG_D2_UNARY(log10)
AG_D2_UNARY(tan)
AG_D2_UNARY(asin)
AG_D2_UNARY(acos)
AG_D2_UNARY(atan)
AG_D2_UNARY(tanh)
AG_D2_UNARY(sinh)
AG_D2_UNARY(cosh)
AG_D2_UNARY(floor)
AG_D2_UNARY(ceil)
AG_D2_UNARY(trunc)
AG_D2_UNARY(cbrt)
AG_D2_UNARY(erf)
AG_D2_BINARY(pow)
AG_D2_BINARY(min)
AG_D2_BINARY(max)
AG_D2_BINARY(atan2)
AG_D2_BINARY(hypot)
#undef AG_D2_UNARY
#undef AG_D2_BINARY
#define AG_N64_USE(NAME)                                                              \
    __device__ __forceinline__ double f_##NAME(double x) { return n64::NAME(x); }     \
    __device__ __forceinline__ d2 f2_##NAME(d2 x) { return n64::NAME(x); }
AG_N64_USE(sqrt)
AG_N64_USE(rsqrt)
AG_N64_USE(exp)
AG_N64_USE(log)
AG_N64_USE(log1p)
__device__ __forceinline__ double rn_div(double x, double y) { return n64::div(x, y); }
__device__ __forceinline__ d2 rn_div(d2 x, d2 y) { return n64::div(x, y); }
__device__ __forceinline__ d2 draw01(double*, ag_u64 seed, ag_u32 g, ag_u32 h, ag_u32 c) {
    return d2{u01_f64(philox_block(seed, g, c).x), u01_f64(philox_block(seed, h, c).x)};
}
#endif

}  // namespace ag
