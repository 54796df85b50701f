// ag_emu64.cuh -- FP64 expression math on the FP32 and integer pipes.
//
// Included by generated kernels lowered with math = 1, 2 or 3, and by native ones
// through ag_tf64.cuh. On GB300 the FP64 pipe
// issues about 1.6 operations per clock per SM against about 110 FFMA and 59
// IMAD (double <-> float conversions run on the FP64 pipe as well), so an
// FP64 expression kernel with transcendental nodes is bound by that pipe long
// before HBM. Here every double is split into a double-float pair
// (hi + lo, two floats, about 48 significant bits) with integer operations,
// the expression is evaluated in double-float arithmetic, and each output is
// reassembled into a double: with one FP64 addition (to_double) where a
// transcendental node hides it, in integers (out_double) elsewhere.
//
// Accuracy: relative error about 2^-46 per function (a few tens of double
// ulps in the worst case), against 2^-53 for the native pipe. Samples whose
// inputs leave [2^-50, 2^60] in magnitude, whose products or quotients fall
// below 2^-102 (where the pair's error terms would be subnormal), whose exp
// arguments leave (-70, 87), whose trig arguments reach 2^24, or whose
// outputs are not finite normal values above 2^-90 are recomputed by the
// generated code with native FP64 (the fallback path), so range, special
// values and large-argument reduction keep FP64 semantics.
//
// Methods (all from the published literature, constants computed by
// gen_emu64_tables.py): Knuth two-sum, Dekker fast-two-sum, FMA two-product;
// double-word addition/multiplication of Joldes, Muller & Popescu (2017);
// Newton-Raphson square root and reciprocal square root from a hardware seed;
// table-driven exp (Tang 1989) and log (Tang 1990); Cody-Waite reduction by
// pi/2 with a 1/32-spaced sine/cosine table; Box-Muller from exact integer
// uniforms.
#pragma once

#include "ag_emu64_tables.cuh"

namespace ag {
namespace e64 {

// Two floats in a register pair, one sample each: add, sub, mul and fma of
// both are one instruction on sm_103a (f32x2). The FP32 lanes are no faster
// that way (59 such instructions a clock and SM against 110 scalar ones), but
// each takes one issue slot in place of two and half the code, and issue is
// what these kernels are bound by. Every function below that does arithmetic
// is a template over F = float or f2 (those with a plain double-float form of
// the same name end in _t); both give the same bits.
struct f2 {
    ag_u64 v;
};
struct b2 {   // a flag per sample
    bool a, b;
};
struct i2 {
    int a, b;
};
struct d2 {
    double a, b;
};
__device__ __forceinline__ f2 pk(float a, float b) {
    f2 r;
#ifdef __CUDA_ARCH__
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
#else
    r.v = ((ag_u64)(unsigned)__float_as_int(b) << 32) | (unsigned)__float_as_int(a);
#endif
    return r;
}
__device__ __forceinline__ float ln0(f2 x) { return __int_as_float((int)(unsigned)x.v); }
__device__ __forceinline__ float ln1(f2 x) { return __int_as_float((int)(unsigned)(x.v >> 32)); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float fneg(float a) { return -a; }
#if defined(__CUDACC__) || defined(__CUDACC_RTC__)
// The assembler joins an f32x2 multiplication with the addition that reads it
// into one fma, .rn or not, which no error-free transformation survives. A
// product is therefore an fma with a -0 that it cannot know, from constant
// memory: a b + (-0) rounds to a b, signed zeros included.
static __constant__ ag_u64 kMinusZeros = 0x8000000080000000ull;
#endif
#ifdef __CUDA_ARCH__
__device__ __forceinline__ f2 fadd(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 fsub(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 fmul(f2 a, f2 b) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(kMinusZeros));
    return r;
}
__device__ __forceinline__ f2 ffma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
#else
__device__ __forceinline__ f2 fadd(f2 a, f2 b) { return pk(fadd(ln0(a), ln0(b)), fadd(ln1(a), ln1(b))); }
__device__ __forceinline__ f2 fsub(f2 a, f2 b) { return pk(fsub(ln0(a), ln0(b)), fsub(ln1(a), ln1(b))); }
__device__ __forceinline__ f2 fmul(f2 a, f2 b) { return pk(fmul(ln0(a), ln0(b)), fmul(ln1(a), ln1(b))); }
__device__ __forceinline__ f2 ffma(f2 a, f2 b, f2 c) {
    return pk(ffma(ln0(a), ln0(b), ln0(c)), ffma(ln1(a), ln1(b), ln1(c)));
}
#endif
__device__ __forceinline__ f2 fneg(f2 a) { return pk(-ln0(a), -ln1(a)); }
template <class F>
struct lanes;
template <>
struct lanes<float> {
    typedef bool flag;
    typedef int whole;
    static __device__ __forceinline__ float bc(float c) { return c; }
};
template <>
struct lanes<f2> {
    typedef b2 flag;
    typedef i2 whole;
    static __device__ __forceinline__ f2 bc(float c) { return pk(c, c); }
};
template <class F>
__device__ __forceinline__ F bc(float c) {   // one constant for every sample
    return lanes<F>::bc(c);
}

template <class F>
struct dfT {
    F hi, lo;
};
typedef dfT<float> df;
typedef dfT<f2> df2;

template <class F>
__device__ __forceinline__ dfT<F> mk(F h, F l) {
    dfT<F> r;
    r.hi = h;
    r.lo = l;
    return r;
}
__device__ __forceinline__ df2 pair(df a, df b) { return mk(pk(a.hi, b.hi), pk(a.lo, b.lo)); }
__device__ __forceinline__ df ln0(df2 x) { return mk(ln0(x.hi), ln0(x.lo)); }
__device__ __forceinline__ df ln1(df2 x) { return mk(ln1(x.hi), ln1(x.lo)); }

// One 16-byte table entry (the packed (hi, lo, hi, lo) rows of the tables).
struct f4 {
    float x, y, z, w;
};
__device__ __forceinline__ f4 ld4(const float* tab, int row) {
#ifdef __CUDA_ARCH__
    const float4 v = __ldg(reinterpret_cast<const float4*>(tab) + row);
    return f4{v.x, v.y, v.z, v.w};
#else
    const float* p = tab + 4 * row;
    return f4{p[0], p[1], p[2], p[3]};
#endif
}

// ---------------------------------------------------------------------------
// Error-free transformations.
// ---------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ dfT<F> two_sum(F a, F b) {
    const F s = fadd(a, b);
    const F bb = fsub(s, a);
    const F e = fadd(fsub(a, fsub(s, bb)), fsub(b, bb));
    return mk(s, e);
}
// Requires |a| >= |b| or a == 0.
template <class F>
__device__ __forceinline__ dfT<F> fast_two_sum(F a, F b) {
    const F s = fadd(a, b);
    const F e = fsub(b, fsub(s, a));
    return mk(s, e);
}
template <class F>
__device__ __forceinline__ dfT<F> two_prod(F a, F b) {
    const F p = fmul(a, b);
    const F e = ffma(a, b, fneg(p));
    return mk(p, e);
}

// ---------------------------------------------------------------------------
// Double-float arithmetic.
// ---------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ dfT<F> neg(dfT<F> x) { return mk(fneg(x.hi), fneg(x.lo)); }

// Accurate sum, relative error <= 3u^2 even under cancellation.
template <class F>
__device__ __forceinline__ dfT<F> add(dfT<F> x, dfT<F> y) {
    const dfT<F> s = two_sum(x.hi, y.hi);
    const dfT<F> t = two_sum(x.lo, y.lo);
    const F c = fadd(s.lo, t.hi);
    const dfT<F> v = fast_two_sum(s.hi, c);
    const F w = fadd(t.lo, v.lo);
    return fast_two_sum(v.hi, w);
}
template <class F>
__device__ __forceinline__ dfT<F> sub(dfT<F> x, dfT<F> y) { return add(x, neg(y)); }
// Sum of terms that cannot cancel (same sign, or |y| well below |x|).
template <class F>
__device__ __forceinline__ dfT<F> add_fast(dfT<F> x, dfT<F> y) {
    const dfT<F> s = two_sum(x.hi, y.hi);
    const F v = fadd(fadd(x.lo, y.lo), s.lo);
    return fast_two_sum(s.hi, v);
}
// The same sum left unnormalised, for a value whose only reader is the
// reassembly into a double (which rounds hi + lo once either way).
template <class F>
__device__ __forceinline__ dfT<F> add_fast_u(dfT<F> x, dfT<F> y) {
    const dfT<F> s = two_sum(x.hi, y.hi);
    return mk(s.hi, fadd(fadd(x.lo, y.lo), s.lo));
}
template <class F>
__device__ __forceinline__ dfT<F> add(dfT<F> x, F y) {
    const dfT<F> s = two_sum(x.hi, y);
    const F v = fadd(x.lo, s.lo);
    return fast_two_sum(s.hi, v);
}
template <class F>
__device__ __forceinline__ dfT<F> mul(dfT<F> x, dfT<F> y) {
    const dfT<F> c = two_prod(x.hi, y.hi);
    const F tl0 = fmul(x.lo, y.lo);
    const F tl1 = ffma(x.hi, y.lo, tl0);
    const F cl2 = ffma(x.lo, y.hi, tl1);
    return fast_two_sum(c.hi, fadd(c.lo, cl2));
}
template <class F>
__device__ __forceinline__ dfT<F> mul(dfT<F> x, F y) {
    const dfT<F> c = two_prod(x.hi, y);
    return fast_two_sum(c.hi, ffma(x.lo, y, c.lo));
}
template <class F>
__device__ __forceinline__ dfT<F> sqr(dfT<F> x) {
    const dfT<F> c = two_prod(x.hi, x.hi);
    return fast_two_sum(c.hi, ffma(fadd(x.hi, x.hi), x.lo, c.lo));
}
// Products whose only consumer is a sum: the same pair before the final
// Fast2Sum (|lo| up to about one ulp of hi), which every sum below accepts.
template <class F>
__device__ __forceinline__ dfT<F> mul_u(dfT<F> x, dfT<F> y) {
    const dfT<F> c = two_prod(x.hi, y.hi);
    const F tl0 = fmul(x.lo, y.lo);
    const F tl1 = ffma(x.hi, y.lo, tl0);
    const F cl2 = ffma(x.lo, y.hi, tl1);
    return mk(c.hi, fadd(c.lo, cl2));
}
template <class F>
__device__ __forceinline__ dfT<F> mul_u(dfT<F> x, F y) {
    const dfT<F> c = two_prod(x.hi, y);
    return mk(c.hi, ffma(x.lo, y, c.lo));
}
template <class F>
__device__ __forceinline__ dfT<F> sqr_u(dfT<F> x) {
    const dfT<F> c = two_prod(x.hi, x.hi);
    return mk(c.hi, ffma(fadd(x.hi, x.hi), x.lo, c.lo));
}
// Products and quotients below 2^-102 in magnitude: the exact error terms
// of the pair arithmetic would be subnormal, so the pair loses precision.
// The lane is flagged for the native path instead.
#define AG_DF_MIN 1.9721522630525295e-31f   // 2^-102
__device__ __forceinline__ df ck(df v, bool& ok) {
    ok = ok && fabsf(v.hi) >= AG_DF_MIN;
    return v;
}
__device__ __forceinline__ df2 ck(df2 v, b2& ok) {
    ok.a = ok.a && fabsf(ln0(v.hi)) >= AG_DF_MIN;
    ok.b = ok.b && fabsf(ln1(v.hi)) >= AG_DF_MIN;
    return v;
}
// Scale by an exact power of two.
template <class F>
__device__ __forceinline__ dfT<F> scale(dfT<F> x, F p2) { return mk(fmul(x.hi, p2), fmul(x.lo, p2)); }
// Sum where the first term dominates: |x.hi| >= |y.hi| (or x == 0), so the
// leading sum is exact by Fast2Sum (Dekker 1971) without the six-operation
// two-sum; the error is that of add_fast. Used where the caller's argument
// ranges prove the ordering.
template <class F>
__device__ __forceinline__ dfT<F> add_quick(dfT<F> x, dfT<F> y) {
    const dfT<F> s = fast_two_sum(x.hi, y.hi);
    const F v = fadd(fadd(x.lo, y.lo), s.lo);
    return fast_two_sum(s.hi, v);
}
template <class F>
__device__ __forceinline__ dfT<F> add_quick(dfT<F> x, F y) {
    const dfT<F> s = fast_two_sum(x.hi, y);
    return fast_two_sum(s.hi, fadd(x.lo, s.lo));
}

// Hardware seeds (MUFU). The host branch exists only so the double-float
// algorithms can be checked by a host build of this header.
__device__ __forceinline__ float rcp_approx(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / x;
#endif
}
__device__ __forceinline__ float rsqrt_approx(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / sqrtf(x);
#endif
}

__device__ __forceinline__ f2 rcp_approx(f2 x) { return pk(rcp_approx(ln0(x)), rcp_approx(ln1(x))); }
__device__ __forceinline__ f2 rsqrt_approx(f2 x) { return pk(rsqrt_approx(ln0(x)), rsqrt_approx(ln1(x))); }

// Reciprocal: FP32 seed refined by two double-float Newton steps.
template <class F>
__device__ __forceinline__ dfT<F> recip_t(dfT<F> y) {
    F r = rcp_approx(y.hi);
    r = ffma(r, ffma(fneg(y.hi), r, bc<F>(1.0f)), r);
    // e = 1 - y*r, computed exactly enough in double-F
    const dfT<F> yr = mul(y, r);
    const F e = fsub(fsub(bc<F>(1.0f), yr.hi), yr.lo);
    return fast_two_sum(r, fmul(r, e));
}
__device__ __forceinline__ df recip(df y) { return recip_t(y); }
// x / y: a float quotient q1 from a twice-refined reciprocal, then one
// correction from the residual x - y q1, formed exactly enough: y.hi q1 =
// p.hi + p.lo (two_prod), x.hi - p.hi is exact (Sterbenz: q1 is within 2^-23
// of the quotient) and the small terms join by fma.
template <class F>
__device__ __forceinline__ dfT<F> div(dfT<F> x, dfT<F> y) {
    F r = rcp_approx(y.hi);
    r = ffma(r, ffma(fneg(y.hi), r, bc<F>(1.0f)), r);
    r = ffma(r, ffma(fneg(y.hi), r, bc<F>(1.0f)), r);   // twice: q1 within ~2^-24, so e's roundings stay at 2^-48 of q
    const F q1 = fmul(x.hi, r);
    const dfT<F> p = two_prod(y.hi, q1);
    F e = fsub(x.hi, p.hi);
    e = fsub(e, p.lo);
    e = fadd(e, x.lo);
    e = ffma(fneg(y.lo), q1, e);
    return fast_two_sum(q1, fmul(e, r));
}

__device__ __forceinline__ bool gt(df a, df b) { return a.hi > b.hi || (a.hi == b.hi && a.lo > b.lo); }
__device__ __forceinline__ bool lt(df a, df b) { return gt(b, a); }
__device__ __forceinline__ bool ge(df a, df b) { return !lt(a, b); }
__device__ __forceinline__ bool le(df a, df b) { return !gt(a, b); }
__device__ __forceinline__ bool eq(df a, df b) { return a.hi == b.hi && a.lo == b.lo; }
__device__ __forceinline__ bool ne(df a, df b) { return !eq(a, b); }
#define AG_E64_CMP2(NAME) \
    __device__ __forceinline__ b2 NAME(df2 x, df2 y) { return b2{NAME(ln0(x), ln0(y)), NAME(ln1(x), ln1(y))}; }
AG_E64_CMP2(gt)
AG_E64_CMP2(lt)
AG_E64_CMP2(ge)
AG_E64_CMP2(le)
AG_E64_CMP2(eq)
AG_E64_CMP2(ne)
#undef AG_E64_CMP2
__device__ __forceinline__ df2 sel(b2 c, df2 x, df2 y) {
    return pair(c.a ? ln0(x) : ln0(y), c.b ? ln1(x) : ln1(y));
}

// ---------------------------------------------------------------------------
// double <-> double-float, with integer operations only (no F2F).
// ---------------------------------------------------------------------------
// |x| in [2^-50, 2^60]: the input range of the double-float path. Squares and
// products of two inputs then stay within [2^-100, 2^120], where the exact
// error terms of the pair arithmetic are still normal floats (the generator
// checks every product it cannot prove to stay above 2^-102).
__device__ __forceinline__ bool in_range(double x) {
    const unsigned ah = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return ah - (973u << 20) <= (111u << 20) - 1u;
}
// The split of a double, and its range test (the flag is cleared when |x|
// leaves [2^-50, 2^60]) from the same integer work: the float exponent of the
// head is the double's less 896, the tail's scale 2^(e-1075) is the head's
// exponent field less 52 (with the sign carried along).
__device__ __forceinline__ df from_double_ck(double x, bool& ok) {
    const unsigned h32 = (unsigned)__double2hiint(x);
    const unsigned l32 = (unsigned)__double2loint(x);
    const unsigned t = (h32 & 0x7fffffffu) - (896u << 20);
    ok = ok && t - (77u << 20) <= (111u << 20) - 1u;
    // hi: the top 24 significant bits (truncated), re-biased to float
    const unsigned hb = __funnelshift_l(l32, t, 3) | (h32 & 0x80000000u);
    // lo: the remaining 29 bits, rounded to a float and scaled by +-2^(ex-1075);
    // |lo| < ulp(hi), so the pair is used without renormalising
    const float lo = __fmul_rn(__uint2float_rn(l32 & 0x1fffffffu), __int_as_float((hb & 0xff800000u) - (52u << 23)));
    return mk(__int_as_float(hb), lo);
}
// Both samples of a lane pair.
__device__ __forceinline__ df2 from_double_ck(double x, double y, b2& ok) {
    return pair(from_double_ck(x, ok.a), from_double_ck(y, ok.b));
}
__device__ __forceinline__ df from_double(double x) {
    bool ok = true;
    return from_double_ck(x, ok);
}
// A normal float (or zero) as a double.
__device__ __forceinline__ double f2d(float f) {
    const unsigned b = (unsigned)__float_as_int(f);
    const unsigned e = (b >> 23) & 0xffu;
    const unsigned hi = (b & 0x80000000u) | ((e + 896u) << 20) | ((b & 0x7fffffu) >> 3);
    const double d = __hiloint2double((int)hi, (int)(b << 29));
    return e == 0u ? 0.0 : d;
}
// The reassembly uses the hardware float->double conversion: two FP64-pipe
// instructions instead of a dozen integer ones on the busier FP32/INT pipes
// (the FP64 pipe has room for a few operations per element at these rates).
__device__ __forceinline__ double to_double(df v) { return __dadd_rn((double)v.hi, (double)v.lo); }
// A result that reassembles exactly: finite, normal and away from underflow.
__device__ __forceinline__ bool out_ok(df v) {
    const unsigned e = ((unsigned)__float_as_int(v.hi) >> 23) & 0xffu;
    return e - 37u <= 216u;   // |hi| in [2^-90, 2^127)
}
__device__ __forceinline__ bool all_of(bool x) { return x; }
__device__ __forceinline__ bool all_of(b2 x) { return x.a && x.b; }
__device__ __forceinline__ bool both_of(bool x, bool y) { return x && y; }
__device__ __forceinline__ b2 both_of(b2 x, b2 y) { return b2{x.a && y.a, x.b && y.b}; }
__device__ __forceinline__ b2 out_ok(df2 v) { return b2{out_ok(ln0(v)), out_ok(ln1(v))}; }
__device__ __forceinline__ d2 to_double(df2 v) { return d2{to_double(ln0(v)), to_double(ln1(v))}; }
// 0 < w < 2^54 as a double-float: the top 24 significant bits exactly, the
// rest rounded once (2^-48 relative).
__device__ __forceinline__ df from_u64(ag_u64 w) {
    const int sh = 40 - __clzll((long long)w);   // bits below the leading 24
    if (sh <= 0) return mk(__uint2float_rn((ag_u32)w), 0.0f);
    const float h = __fmul_rn(__uint2float_rn((ag_u32)(w >> sh)), __int_as_float((sh + 127) << 23));
    const float l = __uint2float_rn((ag_u32)(w & ((1ull << sh) - 1ull)));
    return fast_two_sum(h, l);
}
__device__ __forceinline__ float p2f(int k) { return __int_as_float((k + 127) << 23); }   // 2^k, |k| <= 126
__device__ __forceinline__ f2 p2f(i2 k) { return pk(p2f(k.a), p2f(k.b)); }
// Round to nearest integer for |x| < 2^22 with one FP32 add (no conversion unit).
template <class F>
__device__ __forceinline__ F rint_f(F x) {
    return fsub(fadd(x, bc<F>(12582912.0f)), bc<F>(12582912.0f));
}
__device__ __forceinline__ int rint_i(float x) { return __float_as_int(__fadd_rn(x, 12582912.0f)) - 0x4B400000; }
__device__ __forceinline__ i2 rint_i(f2 x) {
    const f2 t = fadd(x, bc<f2>(12582912.0f));
    return i2{__float_as_int(ln0(t)) - 0x4B400000, __float_as_int(ln1(t)) - 0x4B400000};
}
__device__ __forceinline__ float to_f(int j) { return (float)j; }
__device__ __forceinline__ f2 to_f(i2 j) { return pk((float)j.a, (float)j.b); }
__device__ __forceinline__ int plus(int i, int j) { return i + j; }
__device__ __forceinline__ i2 plus(i2 i, i2 j) { return i2{i.a + j.a, i.b + j.b}; }
__device__ __forceinline__ float fabs_(float x) { return fabsf(x); }
__device__ __forceinline__ f2 fabs_(f2 x) { return pk(fabsf(ln0(x)), fabsf(ln1(x))); }
// lo < x < hi
__device__ __forceinline__ void within(float x, float lo, float hi, bool& ok) { ok = ok && x > lo && x < hi; }
__device__ __forceinline__ void within(f2 x, float lo, float hi, b2& ok) {
    within(ln0(x), lo, hi, ok.a);
    within(ln1(x), lo, hi, ok.b);
}

#if defined(__CUDACC__) || defined(__CUDACC_RTC__) || defined(AG_N64_HOST_CHECK)
// ---------------------------------------------------------------------------
// A float and what is left of a value, joined to a double with integer
// operations: the double of x, plus the rest in units of its last place.
// ---------------------------------------------------------------------------
// 2^(52 - DOWN - e) for |x| in [2^e, 2^(e+1)), with x's sign, from x's exponent
// field; twice that where x is a power of two and the rest (of w's sign) leads
// below it, where the double's unit halves. Needs |x| in [2^(-74-DOWN), 2^127).
template <unsigned DOWN = 0>
__device__ __forceinline__ float join_scale(float x, float w) {
    const unsigned xb = (unsigned)__float_as_int(x), wb = (unsigned)__float_as_int(w);
    const bool down = (xb & 0x7fffffu) == 0u && (wb & 0x7fffffffu) != 0u && ((wb ^ xb) >> 31) != 0u;
    return __int_as_float((int)(((down ? 307u - DOWN : 306u - DOWN) << 23) - (xb & 0x7f800000u) + (xb & 0x80000000u)));
}
template <unsigned DOWN = 0>
__device__ __forceinline__ f2 join_scale(f2 x, f2 w) {
    return pk(join_scale<DOWN>(ln0(x), ln0(w)), join_scale<DOWN>(ln1(x), ln1(w)));
}
// The double of x, `off` units further from zero.
__device__ __forceinline__ double join_bits(float x, int off) {
    const unsigned xb = (unsigned)__float_as_int(x);
    const ag_i64 b = (ag_i64)(((ag_u64)((xb & 0x80000000u) | (((xb & 0x7fffffffu) >> 3) + (896u << 20))) << 32) | (xb << 29)) + off;
    return __hiloint2double((int)(b >> 32), (int)b);
}
__device__ __forceinline__ d2 join_bits(f2 x, i2 off) { return d2{join_bits(ln0(x), off.a), join_bits(ln1(x), off.b)}; }
__device__ __forceinline__ int to_int(float x) { return __float2int_rn(x); }
__device__ __forceinline__ i2 to_int(f2 x) { return i2{to_int(ln0(x)), to_int(ln1(x))}; }
// Whether join_bits and join_scale<DOWN> hold for x: |x| in [2^(-74-DOWN), 2^127).
template <unsigned DOWN>
__device__ __forceinline__ bool join_head(float x) {
    const unsigned e = ((unsigned)__float_as_int(x) >> 23) & 0xffu;
    return e - (53u - DOWN) <= 200u + DOWN;
}
template <unsigned DOWN>
__device__ __forceinline__ b2 join_head(f2 x) {
    return b2{join_head<DOWN>(ln0(x)), join_head<DOWN>(ln1(x))};
}
// hi + lo rounded once, as to_double gives it, without the FP64 pipe: its two
// conversions and one addition are 50 clocks a warp there, which alone held the
// large streaming expression at 73 clocks an element and the batched cross
// products, rotations and inverses at 79 % of that pipe. For |hi + lo| in
// [2^-94, 2^127): the scale alone would leave the floats below 2^-75, so 2^20 of
// it is a factor of its own (by sample: as a pair it took the batched kernel
// from 94 to 98 registers, five CTAs to four, 622 to 673 us).
__device__ __forceinline__ int units_20(float x) { return to_int(__fmul_rn(x, 1048576.0f)); }
__device__ __forceinline__ i2 units_20(f2 x) { return i2{units_20(ln0(x)), units_20(ln1(x))}; }
template <class F>
__device__ __forceinline__ auto out_double(dfT<F> v) {
    const dfT<F> n = fast_two_sum(v.hi, v.lo);   // |lo| <= half an ulp of hi: no carry past its binade
    return join_bits(n.hi, units_20(fmul(n.lo, join_scale<20>(n.hi, n.lo))));
}
// r, or the double of x where x is zero or NaN; `ok` is cleared where neither
// that nor `fits` holds.
__device__ __forceinline__ double or_zero_nan(float x, double r, bool fits, bool& ok) {
    const unsigned xb = (unsigned)__float_as_int(x);
    const bool keep = !(x > 0.0f || x < 0.0f);
    ok = ok && (fits || keep);
    return keep ? __hiloint2double((int)((xb & 0x80000000u) | ((xb & 0x7fffffffu) != 0u ? 0x7ff80000u : 0u)), 0) : r;
}
__device__ __forceinline__ d2 or_zero_nan(f2 x, d2 r, b2 fits, b2& ok) {
    return d2{or_zero_nan(ln0(x), r.a, fits.a, ok.a), or_zero_nan(ln1(x), r.b, fits.b, ok.b)};
}
// A plan's output whose bounds keep it in range: zero and NaN (the root of a
// negative number) leave as they are.
template <class F>
__device__ __forceinline__ auto out_bounded(dfT<F> v, typename lanes<F>::flag& ok) {
    const F n = fadd(v.hi, v.lo);
    const typename lanes<F>::flag fits = join_head<20>(n);
    auto r = out_double(v);
    if (!all_of(fits)) r = or_zero_nan(n, r, fits, ok);
    return r;
}
// For values that may have left the range, out_double after this test: the lane
// runs natively where it fails.
template <class F>
__device__ __forceinline__ void out_double_ok(dfT<F> v, typename lanes<F>::flag& ok) {
    ok = both_of(ok, out_ok(mk(fadd(v.hi, v.lo), v.lo)));
}
#endif

// ---------------------------------------------------------------------------
// Square root and reciprocal square root (Newton-Raphson, one double-float
// correction of a refined hardware seed).
// ---------------------------------------------------------------------------
// Hardware rsqrt seed refined once in FMA form to about 2^-24.5:
// y += (y/2) (1 - x y^2), the residual taken from an FMA.
template <class F>
__device__ __forceinline__ F rsqrt_seed(F x) {
    const F y = rsqrt_approx(x);
    const F e = ffma(fneg(fmul(x, y)), y, bc<F>(1.0f));
    return ffma(fmul(bc<F>(0.5f), y), e, y);
}
// x > 0 (no zero, negative or NaN argument can reach it)
template <class F>
__device__ __forceinline__ dfT<F> sqrt_pos_(dfT<F> x) {
    const F y = rsqrt_seed(x.hi);
    const F s = fmul(x.hi, y);
    const dfT<F> p = two_prod(s, s);
    const F r = fadd(fsub(fsub(x.hi, p.hi), p.lo), x.lo);
    return fast_two_sum(s, fmul(r, fmul(bc<F>(0.5f), y)));
}
// Any argument: a negative or NaN one makes the seed NaN and with it the
// pair; zero (where seed times argument is 0 x inf) keeps its own branch.
__device__ __forceinline__ float or_zero(float x, float r) { return x == 0.0f ? 0.0f : r; }
__device__ __forceinline__ f2 or_zero(f2 x, f2 r) { return pk(or_zero(ln0(x), ln0(r)), or_zero(ln1(x), ln1(r))); }
template <class F>
__device__ __forceinline__ dfT<F> sqrt_t(dfT<F> x) {
    const dfT<F> res = sqrt_pos_(x);
    return mk(or_zero(x.hi, res.hi), or_zero(x.hi, res.lo));
}
__device__ __forceinline__ df sqrt_(df x) { return sqrt_t(x); }
template <class F>
__device__ __forceinline__ dfT<F> sqrt_nn_(dfT<F> x) {
    return sqrt_t(x);
}
// One Newton step on a float seed y: e = 1 - x y^2 and rsqrt x = y (1 + e/2).
// y^2 = p + q exactly (two_prod); x.hi p is within 2^-22 of 1, so fma(-x.hi,
// p, 1) carries e to 2^-24 of itself and the two smaller products join it by
// fma; the correction y e / 2 is ~2^-23 of y, so the result is good to ~2^-47.
template <class F>
__device__ __forceinline__ dfT<F> rsqrt_t(dfT<F> x) {
    const F y = rsqrt_seed(x.hi);
    const dfT<F> yy = two_prod(y, y);
    F e = ffma(fneg(x.hi), yy.hi, bc<F>(1.0f));
    e = ffma(fneg(x.hi), yy.lo, e);
    e = ffma(fneg(x.lo), yy.hi, e);
    // x.hi <= 0, NaN or +inf make the seed or the residual NaN, so the pair is
    // NaN there without a test (and such lanes take the native path)
    return fast_two_sum(y, fmul(fmul(y, e), bc<F>(0.5f)));
}
__device__ __forceinline__ df rsqrt_(df x) { return rsqrt_t(x); }

// ---------------------------------------------------------------------------
// exp: x = (64k + j) ln2/64 + r, |r| <= ln2/128; e^x = 2^k 2^(j/64) e^r.
// ---------------------------------------------------------------------------
// The flag is cleared outside -70 < x < 87, where 2^k leaves the float range
// or the result's low part would be subnormal (the native lane computes it).
__device__ __forceinline__ df exp_table(int m) {
    const int j = m & 63;
    return mk(__ldg(&kExp2TabHi[j]), __ldg(&kExp2TabLo[j]));
}
__device__ __forceinline__ df2 exp_table(i2 m) { return pair(exp_table(m.a), exp_table(m.b)); }
__device__ __forceinline__ int exp_power(int m) {
    const int k = m >> 6;
    return k < -126 ? -126 : (k > 126 ? 126 : k);
}
__device__ __forceinline__ i2 exp_power(i2 m) { return i2{exp_power(m.a), exp_power(m.b)}; }
template <class F>
__device__ __forceinline__ dfT<F> exp_(dfT<F> x, typename lanes<F>::flag& ok) {
    within(x.hi, -70.0f, 87.0f, ok);
    const F mx = fmul(x.hi, bc<F>(AG_INV_LN2_64));
    const F mf = rint_f(mx);
    const typename lanes<F>::whole m = rint_i(mx);
    const F r1 = ffma(fneg(mf), bc<F>(AG_LN2_64_1), x.hi);   // exact (Sterbenz)
    dfT<F> r = two_sum(r1, x.lo);
    r = sub(r, two_prod(mf, bc<F>(AG_LN2_64_2)));
    r = add(r, fmul(fneg(mf), bc<F>(AG_LN2_64_3)));
    // e^r - 1 = r + r^2/2 + r^3 (1/6 + r/24 + r^2/120)
    const F rh = r.hi;
    const F tail = fmul(fmul(rh, fmul(rh, rh)),
                        ffma(rh, ffma(rh, bc<F>(8.33333333e-3f), bc<F>(4.16666667e-2f)), bc<F>(1.66666667e-1f)));
    // |r| <= ln2/128, so each sum below is led by its first term
    dfT<F> p = add_quick(r, scale(sqr(r), bc<F>(0.5f)));
    p = add_quick(p, tail);
    const dfT<F> T = exp_table(m);
    const dfT<F> res = add_quick(T, mul(T, p));
    return scale(res, p2f(exp_power(m)));
}

// ---------------------------------------------------------------------------
// log: y = 2^e m, m in [0.75, 1.5), i = round(128 (m - 1)), c_i ~ 1/(1 + i/128)
// (c_0 = 1), t = y 2^-e c_i - 1 (|t| < 2^-7), log y = e ln2 - log c_i + log(1+t).
// log_s(s, x) is log(s + x) for s in {0, 1}: log for s = 0, log1p for s = 1,
// with t formed from s and x separately so 1 + x is never rounded.
// ---------------------------------------------------------------------------
// log(1+t) for |t| <= 2^-10.6: t - t^2/2 in double-float, the rest
// t^2 (t/3 - t^2/4 + t^3/5) in float (at most 2^-47.6 relative to t).
template <class F>
__device__ __forceinline__ dfT<F> log1p_poly(dfT<F> t) {
    // h = -t^2/2 as an unnormalised pair: -t.hi^2/2 rounded, its exact error
    // and -t.hi t.lo; r = t^2 q = (hh + hl) (-2 q), the -2 folded into q (r
    // needs t^2 to F accuracy, so the t.lo part of h joins it)
    const F th = t.hi;
    const F u = fmul(bc<F>(-0.5f), th);   // exact
    const F hh = fmul(th, u);
    const F hl = ffma(fneg(th), t.lo, ffma(th, u, fneg(hh)));
    const F r = fmul(fadd(hh, hl),
                              fmul(th, ffma(th, ffma(th, bc<F>(-0.4f), bc<F>(0.5f)), bc<F>(-0.666666667f))));
    return add_quick(add_quick(t, mk(hh, hl)), r);
}
// log_s(s, x) for s + x > 0 with 2^-120 < s + x < 2^120 known in advance
// (checked = false) skips the validity test. MODE selects how the reduced
// argument t = s A - 1 + x A is formed: 0 for log (s = 0: x.hi A is within
// 2^-10 of 1, so x.hi A - 1 is exact by Sterbenz), 1 for log1p (s = 1:
// A - 1 as an exact two-sum), 2 for s in {0, 1} at run time where s A - 1 is
// a single exact FMA (s = 1 only with 1/2 <= s + x < 1, A in [2/3, 2]).
enum { LOG_S0 = 0, LOG_S1 = 1, LOG_SRT = 2 };
// The integer part of the reduction: A = c_i 2^-e, -log c_i and e ln2 from the
// tables, and whether y was positive with an exponent they cover.
struct log_row {
    float A, Lh, Ll, Eh, El;
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
    const int i = rint_i(__fmaf_rn(m, 1024.0f, -1024.0f)) + AG_LOG_TAB_OFF;   // (m - 1) 1024, exact
    const f4 cl = ld4(kLogCL, i);
    log_row r;
    r.A = __int_as_float((int)((unsigned)__float_as_int(cl.x) - ((unsigned)e << 23)));   // c 2^-e, exact for valid e
    r.Lh = cl.y;
    r.Ll = cl.z;
    // e ln2 from a table covering every e the bits above can give (out-of-range
    // e is flagged below)
    const int ei = e + AG_LN2_TAB_OFF;
#ifdef __CUDA_ARCH__
    const float2 ep = __ldg(reinterpret_cast<const float2*>(kLn2Mul) + ei);
    r.Eh = ep.x;
    r.El = ep.y;
#else
    r.Eh = kLn2Mul[2 * ei];
    r.El = kLn2Mul[2 * ei + 1];
#endif
    r.valid = yh > 0.0f && e > -120 && e < 120;
    return r;
}
template <class F>
struct log_rows {
    F A;
    dfT<F> L, E;
    typename lanes<F>::flag valid;
};
__device__ __forceinline__ log_rows<float> log_tables(float yh) {
    const log_row r = log_reduce(yh);
    return log_rows<float>{r.A, mk(r.Lh, r.Ll), mk(r.Eh, r.El), r.valid};
}
__device__ __forceinline__ log_rows<f2> log_tables(f2 yh) {
    const log_row r = log_reduce(ln0(yh)), s = log_reduce(ln1(yh));
    return log_rows<f2>{pk(r.A, s.A), mk(pk(r.Lh, s.Lh), pk(r.Ll, s.Ll)), mk(pk(r.Eh, s.Eh), pk(r.El, s.El)),
                        b2{r.valid, s.valid}};
}
__device__ __forceinline__ df or_nan(bool ok, df v) { return ok ? v : mk(__int_as_float(0x7fc00000), 0.0f); }
__device__ __forceinline__ df2 or_nan(b2 ok, df2 v) { return pair(or_nan(ok.a, ln0(v)), or_nan(ok.b, ln1(v))); }

template <bool checked = true, int MODE = LOG_S1, class F>
__device__ __forceinline__ dfT<F> log_s(F s, dfT<F> x) {
    const log_rows<F> R = log_tables(fadd(s, x.hi));
    const F A = R.A;
    // x A = p + (x.lo A + p.lo), the pair left unnormalised for the sum
    const dfT<F> p = two_prod(x.hi, A);
    const F pl = ffma(x.lo, A, p.lo);
    dfT<F> t;
    if (MODE == LOG_S0) {
        t = fast_two_sum(fsub(p.hi, bc<F>(1.0f)), pl);
    } else if (MODE == LOG_SRT) {
        const dfT<F> u = two_sum(ffma(s, A, bc<F>(-1.0f)), p.hi);
        t = fast_two_sum(u.hi, fadd(pl, u.lo));
    } else {
        // B = A - 1 exactly; B.lo = 0 whenever B and x A can cancel (c_i - 1
        // is exact by Sterbenz for e = 0), so t keeps 2^-48 of itself there;
        // for e != 0 the result is >= 0.29 in magnitude and an error of 2^-48
        // of the terms is 2^-46.5 of it
        const dfT<F> B = two_sum(A, bc<F>(-1.0f));
        const dfT<F> u = two_sum(B.hi, p.hi);
        t = fast_two_sum(u.hi, fadd(fadd(B.lo, pl), u.lo));
    }
    // |E| >= ln2 > |L + log1p(t)| except for e == 0 (E = 0), |L| >= 2^-10.6
    // >= |t| except for i == 0 (L = 0): each sum is led by its first term.
    dfT<F> res;
    if (MODE == LOG_SRT) {
        // The Box-Muller logarithm (halved again by the square root that
        // follows): one chain E + L + t + h, h = -t^2/2 as an unnormalised
        // pair, with every low part and r = t^2 (t/3 - t^2/4 + t^3/5) gathered
        // into one float. About a quarter of the operations of the two
        // renormalised sums below, at a few per cent more mean error.
        const F th = t.hi;
        const F uu = fmul(bc<F>(-0.5f), th);
        const F hh = fmul(th, uu);
        const F hl = ffma(fneg(th), t.lo, ffma(th, uu, fneg(hh)));
        const F r = fmul(fadd(hh, hl),
                         fmul(th, ffma(th, ffma(th, bc<F>(-0.4f), bc<F>(0.5f)), bc<F>(-0.666666667f))));
        const dfT<F> a1 = fast_two_sum(R.E.hi, R.L.hi);
        const dfT<F> a2 = fast_two_sum(a1.hi, th);
        const dfT<F> a3 = fast_two_sum(a2.hi, hh);   // |h| <= 2^-11.6 |t|
        const F lo = fadd(fadd(fadd(fadd(a1.lo, a2.lo), fadd(a3.lo, R.E.lo)), fadd(R.L.lo, t.lo)), fadd(hl, r));
        res = fast_two_sum(a3.hi, lo);
    } else {
        res = add_quick(R.E, add_quick(R.L, log1p_poly(t)));
    }
    return checked ? or_nan(R.valid, res) : res;
}
template <class F>
__device__ __forceinline__ dfT<F> log_t(dfT<F> x) {
    return log_s<true, LOG_S0>(bc<F>(0.0f), x);
}
template <class F>
__device__ __forceinline__ dfT<F> log1p_t(dfT<F> x) {
    return log_s<true, LOG_S1>(bc<F>(1.0f), x);
}
__device__ __forceinline__ df log_(df x) { return log_t(x); }
__device__ __forceinline__ df log1p_(df x) { return log1p_t(x); }
// log1p of an argument known to be >= 0 and below 2^60 (an input in the
// double-float range, or an expression of such inputs that cannot grow past it)
template <class F>
__device__ __forceinline__ dfT<F> log1p_nn_(dfT<F> x) {
    return log_s<false, LOG_S1>(bc<F>(1.0f), x);
}

// ---------------------------------------------------------------------------
// sin/cos: r in [-pi/4, pi/4] (a little beyond is fine) split as r = j/2048 + t
// with |t| <= 2^-12; with S_j, C_j = sin, cos(j/2048) from a table,
// sin r = S_j (1 + cm1) + C_j st and cos r = C_j (1 + cm1) - S_j st, where
// st = sin t = t + t^3 (-1/6 + t^2/120) and cm1 = cos t - 1 = t^2 (-1/2 + t^2/24).
// For |t| <= 2^-12 the cubic and quadratic terms are below 2^-26.6 of t and of
// 1, so they are computed in float from t.hi; only t and the products with
// the table values are double-float.
// ---------------------------------------------------------------------------
// One output of sin/cos at x = q pi/2 + r: sin x is +-sin r or +-cos r by
// quadrant, and both are A (1 + cm1) + B st with the table pair (A, B) =
// (S_j, C_j) for sin r and (C_j, -S_j) for cos r, so only the wanted one is
// evaluated.
// The table pair and the sign of the wanted output at quadrant q (cos x = sin(x + pi/2)).
template <class F>
struct trig_rows {
    dfT<F> A, B;
    typename lanes<F>::flag minus;
};
__device__ __forceinline__ trig_rows<float> trig_table(const f4& sc, int q, bool want_cos) {
    const int qq = (q + (want_cos ? 1 : 0)) & 3;
    const bool odd = qq & 1;
    return trig_rows<float>{odd ? mk(sc.z, sc.w) : mk(sc.x, sc.y), odd ? mk(-sc.x, -sc.y) : mk(sc.z, sc.w), (qq & 2) != 0};
}
__device__ __forceinline__ trig_rows<float> trig_table(int j, int q, bool want_cos) {
    return trig_table(ld4(kSinCos2048, j + AG_SC_TAB_OFF), q, want_cos);
}
__device__ __forceinline__ trig_rows<f2> trig_table(i2 j, i2 q, bool want_cos) {
    const trig_rows<float> r = trig_table(j.a, q.a, want_cos), s = trig_table(j.b, q.b, want_cos);
    return trig_rows<f2>{pair(r.A, s.A), pair(r.B, s.B), b2{r.minus, s.minus}};
}
__device__ __forceinline__ df neg_if(bool c, df v) { return c ? neg(v) : v; }
__device__ __forceinline__ df2 neg_if(b2 c, df2 v) { return pair(neg_if(c.a, ln0(v)), neg_if(c.b, ln1(v))); }
// The table step for x = q pi/2 + a + t.
template <class F>
__device__ __forceinline__ dfT<F> trig_tail(const trig_rows<F>& R, dfT<F> t) {
    const F th = t.hi;
    const F th2 = fmul(th, th);
    const F cubic = fmul(fmul(th, th2), ffma(th2, bc<F>(8.33333333e-3f), bc<F>(-1.66666667e-1f)));
    const F cm1 = fmul(th2, ffma(th2, bc<F>(4.16666667e-2f), bc<F>(-0.5f)));
    // |A| >= sin(2^-11) >= 2 |B t| for j != 0, and A = 0 at j = 0 for sin r:
    // the sum is led by A
    const dfT<F> v = add_quick(add_quick(R.A, mul_u(R.B, t)), ffma(R.A.hi, cm1, fmul(R.B.hi, cubic)));
    return neg_if(R.minus, v);
}
__device__ __forceinline__ int clamp_row(int j) {   // NaN-safe index
    return j < -AG_SC_TAB_OFF ? -AG_SC_TAB_OFF : (j > AG_SC_TAB_OFF ? AG_SC_TAB_OFF : j);
}
__device__ __forceinline__ i2 clamp_row(i2 j) { return i2{clamp_row(j.a), clamp_row(j.b)}; }
template <class F>
__device__ __forceinline__ dfT<F> trig_core(dfT<F> r, typename lanes<F>::whole q, bool want_cos) {
    const typename lanes<F>::whole j = clamp_row(rint_i(fmul(r.hi, bc<F>(2048.0f))));
    const dfT<F> t = fast_two_sum(fsub(r.hi, fmul(to_f(j), bc<F>(4.8828125e-4f))), r.lo);   // exact first difference
    return trig_tail(trig_table(j, q, want_cos), t);
}
// Cody-Waite reduction by pi/2; valid for |k| < 4096, flagged otherwise.
__device__ __forceinline__ df dfc(double x);

#ifdef __CUDA_ARCH__
__device__ __forceinline__ ag_u64 umulhi64(ag_u64 a, ag_u64 b) { return __umul64hi(a, b); }
#else
inline ag_u64 umulhi64(ag_u64 a, ag_u64 b) { return (ag_u64)(((unsigned __int128)a * b) >> 64); }
#endif

// Payne-Hanek reduction (Payne & Hanek 1983) of a float h with 6000 <= |h| <
// 2^24, in 64-bit integer arithmetic: |h| = m 2^E with a 24-bit integer m and
// E in [-11, 0]; |h| 2/pi = m W 2^(E-192) with W = 2/pi to 192 bits, so the
// quadrant and 128 fraction bits come out of the three 64x64 products m W_i.
// Returns |h| - k pi/2 (a double-float, |.| <= pi/4) and k.
__device__ __forceinline__ df reduce_ph(float h, int& k, bool& ok) {
    const unsigned b = (unsigned)__float_as_int(h);
    const ag_u64 m = (ag_u64)((b & 0x7fffffu) | 0x800000u);
    int sh = 150 - (int)((b >> 23) & 0xffu);   // -E
    ok = ok && sh >= 0 && sh <= 11;
    sh = sh < 0 ? 0 : (sh > 11 ? 11 : sh);
    // m W from bit 64 up, as (a2:a1:a0)
    const ag_u64 p2h = umulhi64(m, AG_2OPI_W2);
    const ag_u64 p1l = m * AG_2OPI_W1, p1h = umulhi64(m, AG_2OPI_W1);
    const ag_u64 p0l = m * AG_2OPI_W0, p0h = umulhi64(m, AG_2OPI_W0);
    const ag_u64 a0 = p1l + p2h;
    const ag_u64 c0 = a0 < p1l ? 1ull : 0ull;
    ag_u64 a1 = p0l + p1h;
    ag_u64 c1 = a1 < p0l ? 1ull : 0ull;
    a1 += c0;
    c1 += a1 < c0 ? 1ull : 0ull;
    const ag_u64 a2 = p0h + c1;
    // the binary point sits sh bits into a2: integer part, then 128 fraction bits
    ag_u64 ip = a2 >> sh;
    ag_u64 fh = sh ? (a2 << (64 - sh)) | (a1 >> sh) : a1;
    ag_u64 fl = sh ? (a1 << (64 - sh)) | (a0 >> sh) : a0;
    // to the nearest quadrant: a fraction >= 1/2 becomes negative
    const bool up = (fh >> 63) != 0;
    ip += up ? 1ull : 0ull;
    if (up) {
        fl = ~fl + 1ull;
        fh = ~fh + (fl == 0 ? 1ull : 0ull);
    }
    // |fraction| = (fh:fl) 2^-128, normalised: top 48 bits as a double-float
    const int lz = fh ? __clzll((long long)fh) : 64 + __clzll((long long)(fl | 1ull));
    ok = ok && lz < 78;   // |r| >= 2^-78: otherwise too close to k pi/2 for the float exponent range
    const int l = lz < 78 ? lz : 77;
    const ag_u64 top = l < 64 ? (l ? (fh << l) | (fl >> (64 - l)) : fh) : (fl << (l - 64));
    const float th = __fmul_rn(__uint2float_rn((ag_u32)(top >> 40)), p2f(-24 - l));
    const float tl = __fmul_rn(__uint2float_rn((ag_u32)((top >> 16) & 0xffffffu)), p2f(-48 - l));
    df f = fast_two_sum(th, tl);
    f = mul(f, mk(AG_PIO2_HI, AG_PIO2_LO));
    k = (int)(ip & 3ull);
    return up ? neg(f) : f;
}

// |x| < 6000: Cody-Waite in float (three-part pi/2, exact products for |k| <
// 4096); 6000 <= |x| < 2^24: Payne-Hanek in integers; beyond, flagged (the
// native lane reduces it).
template <class F>
__device__ __forceinline__ dfT<F> reduce_cw(dfT<F> x, typename lanes<F>::whole& q) {
    const F kx = fmul(x.hi, bc<F>(AG_TWO_OVER_PI));
    const F kf = rint_f(kx);
    const F r1 = ffma(fneg(kf), bc<F>(AG_PIO2_1), x.hi);
    dfT<F> r = two_sum(r1, x.lo);
    r = sub(r, two_prod(kf, bc<F>(AG_PIO2_2)));
    r = add(r, fmul(fneg(kf), bc<F>(AG_PIO2_3)));
    q = rint_i(kx);
    return r;
}
__device__ __forceinline__ df reduce_(df x, int& q, bool& ok) {
    const float ax = fabsf(x.hi);
    df r;
    if (ax < 6000.0f) {
        r = reduce_cw(x, q);
    } else {
        int k;
        r = reduce_ph(ax, k, ok);
        if (x.hi < 0.0f) {
            r = neg(r);
            k = -k;
        }
        r = add(r, x.lo);   // x - k pi/2 = (hi - k pi/2) + lo
        q = k;
        // |lo| can reach ulp(hi)/2, up to 1/2 below 2^24: bring r back into [-pi/4, pi/4]
        if (r.hi > 0.78539816f) {
            r = sub(r, mk(AG_PIO2_HI, AG_PIO2_LO));
            q += 1;
        } else if (r.hi < -0.78539816f) {
            r = add(r, mk(AG_PIO2_HI, AG_PIO2_LO));
            q -= 1;
        }
    }
    return r;
}
__device__ __forceinline__ df2 reduce_(df2 x, i2& q, b2& ok) {
    if (fabsf(ln0(x.hi)) < 6000.0f && fabsf(ln1(x.hi)) < 6000.0f) return reduce_cw(x, q);
    const df r0 = reduce_(ln0(x), q.a, ok.a);
    return pair(r0, reduce_(ln1(x), q.b, ok.b));
}
template <class F>
__device__ __forceinline__ dfT<F> trig_(dfT<F> x, bool want_cos, typename lanes<F>::flag& ok) {
    typename lanes<F>::whole q;
    const dfT<F> r = reduce_(x, q, ok);
    return trig_core(r, q, want_cos);
}
template <class F>
__device__ __forceinline__ dfT<F> sin_(dfT<F> x, typename lanes<F>::flag& ok) {
    return trig_(x, false, ok);
}
template <class F>
__device__ __forceinline__ dfT<F> cos_(dfT<F> x, typename lanes<F>::flag& ok) {
    return trig_(x, true, ok);
}
// sin(pi v): exact reduction v = q/2 + r, |r| <= 1/4, then sin/cos of pi r.
__device__ __forceinline__ df sinpi_(df v) {
    const float qf = rint_f(__fmul_rn(v.hi, 2.0f));
    const df r = fast_two_sum(__fsub_rn(v.hi, __fmul_rn(qf, 0.5f)), v.lo);
    return trig_core(mul(r, mk(AG_PI_HI, AG_PI_LO)), rint_i(__fmul_rn(v.hi, 2.0f)), false);
}

// ---------------------------------------------------------------------------
// Philox draws as double-floats. Uniform: (2w+1) 2^-33 is exact in a
// double-float, so uniform(lo, hi) fills with power-of-two ranges are
// bit-exact. The normal draw (Box-Muller) is in ag_emu64_bm.cuh, which plans
// with normal leaves include.
// ---------------------------------------------------------------------------
__device__ __forceinline__ df draw01_df(ag_u64 seed, ag_u32 g, ag_u32 c) {
    const ag_u32 w = ag::philox_block(seed, g, c).x;
    return scale(from_u64(2ull * w + 1ull), p2f(-33));
}
__device__ __forceinline__ df2 draw01_df(ag_u64 seed, ag_u32 g, ag_u32 h, ag_u32 c) {
    return pair(draw01_df(seed, g, c), draw01_df(seed, h, c));
}

// ---------------------------------------------------------------------------
// Scalars, simple nodes and the bridge to native FP64 for functions without a
// double-float kernel (each costs FP64-pipe work, like the native plan).
// ---------------------------------------------------------------------------
__device__ __forceinline__ df dfc(double x) {   // any double (runtime scalars, literals)
    const float h = __double2float_rn(x);
    const float l = isfinite(h) ? __double2float_rn(x - (double)h) : 0.0f;
    return mk(h, l);
}
// |x|: |hi|, and lo with the sign of hi taken off
__device__ __forceinline__ df abs_(df x) {
    return mk(fabsf(x.hi), __int_as_float(__float_as_int(x.lo) ^ (__float_as_int(x.hi) & (int)0x80000000)));
}
__device__ __forceinline__ df sign_(df x) {
    return mk(x.hi > 0.0f ? 1.0f : (x.hi < 0.0f ? -1.0f : 0.0f), 0.0f);
}
__device__ __forceinline__ df min_(df a, df b) { return lt(b, a) ? b : a; }
__device__ __forceinline__ df max_(df a, df b) { return gt(b, a) ? b : a; }
__device__ __forceinline__ df2 both(df x) { return pair(x, x); }   // a value all samples share
__device__ __forceinline__ d2 both(double x) { return d2{x, x}; }
__device__ __forceinline__ df2 abs_(df2 x) { return pair(abs_(ln0(x)), abs_(ln1(x))); }
__device__ __forceinline__ df2 sign_(df2 x) { return pair(sign_(ln0(x)), sign_(ln1(x))); }
__device__ __forceinline__ df2 min_(df2 x, df2 y) { return pair(min_(ln0(x), ln0(y)), min_(ln1(x), ln1(y))); }
__device__ __forceinline__ df2 max_(df2 x, df2 y) { return pair(max_(ln0(x), ln0(y)), max_(ln1(x), ln1(y))); }
__device__ __forceinline__ double as_d(df x) { return (double)x.hi + (double)x.lo; }
#define AG_E64_NATIVE1(NAME)                                                                   \
    __device__ __forceinline__ df nat_##NAME(df x) { return dfc(ag::f_##NAME(as_d(x))); }      \
    __device__ __forceinline__ df2 nat_##NAME(df2 x) { return pair(nat_##NAME(ln0(x)), nat_##NAME(ln1(x))); }
#define AG_E64_NATIVE2(NAME)                                                                   \
    __device__ __forceinline__ df nat_##NAME(df a, df b) { return dfc(ag::f_##NAME(as_d(a), as_d(b))); } \
    __device__ __forceinline__ df2 nat_##NAME(df2 x, df2 y) {                                  \
        return pair(nat_##NAME(ln0(x), ln0(y)), nat_##NAME(ln1(x), ln1(y)));                   \
    }
AG_E64_NATIVE1(expm1)
AG_E64_NATIVE1(exp2)
AG_E64_NATIVE1(log2)
AG_E64_NATIVE1(log10)
AG_E64_NATIVE1(tan)
AG_E64_NATIVE1(asin)
AG_E64_NATIVE1(acos)
AG_E64_NATIVE1(atan)
AG_E64_NATIVE1(tanh)
AG_E64_NATIVE1(sinh)
AG_E64_NATIVE1(cosh)
AG_E64_NATIVE1(floor)
AG_E64_NATIVE1(ceil)
AG_E64_NATIVE1(trunc)
AG_E64_NATIVE1(cbrt)
AG_E64_NATIVE1(erf)
AG_E64_NATIVE2(pow)
AG_E64_NATIVE2(atan2)
AG_E64_NATIVE2(hypot)
#undef AG_E64_NATIVE1
#undef AG_E64_NATIVE2

}  // namespace e64
namespace x64 = e64;   // the spelling of a plan's two-sample code
}  // namespace ag
