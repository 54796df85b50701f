// ag_emu64_bm.cuh -- the Box-Muller draw in double-float (N(mu, sigma) and
// lognormal leaves of plans lowered with math = 1), included by the generated
// kernels of plans that draw normals, after ag_emu64.cuh.
//
// z = sqrt(-2 log u) sin(pi v) (random/detail/Backend.h:209-236, first normal
// only) from the reference's own double uniforms u and v, reproduced exactly
// in integers; log(u) is taken as log(u) for u < 1/2 and as log1p(-(1-u))
// above, with 1-u formed in integers; sin(pi v) is reduced in integers to a
// point of a table of sin and pi cos of pi k/4096 over the whole period and an
// exact remainder.
#pragma once

#include "ag_emu64_bm_tables.cuh"

#if defined(__CUDACC__) || defined(__CUDACC_RTC__)
#define AG_NOINLINE __noinline__
#else
#define AG_NOINLINE __attribute__((noinline))
#endif

namespace ag {
namespace e64 {

// sgn w 2^-54 for 0 < w < 2^54: normalised so the leading bit sits at 2^53,
// the top 24 bits exact and the next 30 rounded once (2^-48 relative); the
// pair is left with |lo| < ulp(hi). sgn is the sign bit (0 or 0x80000000).
__device__ AG_NOINLINE df from_u54_2m54_any(ag_u64 w, ag_u32 sgn) {
    const int lz = __clzll((long long)w) - 10;   // 0 .. 53
    const ag_u64 wn = w << lz;                    // [2^53, 2^54)
    const ag_u32 sc = ((ag_u32)(103 - lz) << 23) | sgn;   // +-2^(-24-lz): 2^30 units of wn, times 2^-54
    const float h = __fmul_rn(__uint2float_rn((ag_u32)(wn >> 30)), __int_as_float(sc));
    const float l = __fmul_rn(__uint2float_rn((ag_u32)wn & 0x3fffffffu), __int_as_float(sc - (30u << 23)));
    return mk(h, l);
}
// The same in 32-bit words when w >= 2^32 (all but 2^-22 of the draws: the
// normalising shift stays below 32), the general form out of line otherwise.
// No integer-to-float conversion unit: the head's float is assembled from
// its bits (the top 24 bits of w << lz are its significand, the shift gives
// its exponent), and the tail is the next 23 bits made exact by the 2^23
// exponent trick (one OR and one subtraction) and scaled; the 7 bits below
// are dropped, 2^-47 of u.
__device__ __forceinline__ df from_u54_2m54(ag_u64 w, ag_u32 sgn) {
    const ag_u32 hi = (ag_u32)(w >> 32), lo = (ag_u32)w;
    if (hi == 0u) return from_u54_2m54_any(w, sgn);
    const int lz = __clz((int)hi) - 10;   // 0 .. 21
    const ag_u32 nh = __funnelshift_l(lo, hi, (unsigned)lz), nl = lo << lz;   // w << lz in [2^53, 2^54)
    const ag_u32 top = __funnelshift_l(nl, nh, 2u);                           // bits 53..30, in [2^23, 2^24)
    // top 2^(30 - 54 - lz): exponent -1 - lz, significand top
    const float h = __int_as_float((int)(((ag_u32)(126 - lz) << 23) | (top & 0x7fffffu) | sgn));
    // bits 29..7 as an exact float, weight 2^(7 - 54 - lz)
    const float r = __fsub_rn(__int_as_float((int)(0x4B000000u | ((nl >> 7) & 0x7fffffu))), 8388608.0f);
    const float l = __fmul_rn(r, __int_as_float((int)(((ag_u32)(80 - lz) << 23) | sgn)));
    return mk(h, l);
}

// sin(pi (k/4096 + t)) from the table entry (S, pi C) of k and the exact
// remainder |t| <= 2^-13 in half-turns: with r = pi t, S (1 + cm1) + C st,
// st = sin r = r + r^3 (-1/6 + r^2/120) and cm1 = cos r - 1 = r^2 (-1/2 +
// r^2/24). C r = (pi C) t and C r^3 = (pi C) t r^2, so only the float r of the
// small terms needs pi; the leading product is (pi C) t in double-float.
// |S| >= sin(pi/4096) >= |C r| except where S = 0: the sum is led by S.
template <class F>
__device__ __forceinline__ dfT<F> sin_from_period_table(dfT<F> S, dfT<F> PC, dfT<F> t) {
    const F th = t.hi;
    // r = pi t rounded once (pi's and t's low parts joined by FMA): the
    // quadratic term needs r to float accuracy
    const F rh = ffma(bc<F>(AG_PI_HI), th, ffma(bc<F>(AG_PI_HI), t.lo, fmul(bc<F>(AG_PI_LO), th)));
    const F rh2 = fmul(rh, rh);
    const F cub = fmul(fmul(th, rh2), ffma(rh2, bc<F>(8.33333333e-3f), bc<F>(-1.66666667e-1f)));
    const F cm1 = fmul(rh2, ffma(rh2, bc<F>(4.16666667e-2f), bc<F>(-0.5f)));
    return add_quick(add_quick(S, mul_u(PC, t)), ffma(S.hi, cm1, fmul(PC.hi, cub)));
}

// The integer part of one draw.
struct bm_words {
    float s;        // log(u) = log(s + w)
    df w;
    float fh, fl;   // the remainder of v, in units of 2^-35 and 2^-53 half-turns
    f4 sc;          // (S, pi C) of v's table point
};
__device__ __forceinline__ bm_words bm_draw(ag_u64 seed, ag_u32 g, ag_u32 c) {
    const ag::q4 x = ag::philox_block(seed, g, c);
    bm_words b;
    // u is the reference's double z 2^-53 + 2^-54 (random/detail/Backend.h
    // uniformDoubleHq): exact below 1/2, rounded to even above it, where it is
    // k 2^-53 with k = z + (z & 1). So u = w 2^-54 with w = 2 z + 1 below 1/2,
    // and 1 - u = w 2^-54 with w = 2^54 - 2 k (even, at most 2^53) above it.
    // log(u) for u in [2^-54, 1/2) or log1p(-w) for w in [0, 1/2]; w = 0 (u
    // rounded to 1) gives a zero argument to the square root below, whose NaN
    // sends the lane to the native path
    const ag_u64 z = (ag_u64)x.x ^ ((ag_u64)x.y << 21);
    const bool lower = z < (1ull << 52);
    const ag_u64 w = lower ? 2ull * z + 1ull : (1ull << 54) - 2ull * (z + (z & 1ull));
    b.s = lower ? 0.0f : 1.0f;
    b.w = from_u54_2m54(w, lower ? 0u : 0x80000000u);
    // v is the reference's double zy 2^-52 + 2^-53: exact below 1, rounded to
    // even above it. So v = V 2^-53 with V = 2 zy + 1, or 2 (zy + (zy & 1))
    // for zy >= 2^52, V <= 2^54. In integers: K = round(V / 2^41) in [0, 8192]
    // counts steps of 1/4096 half-turn (the table point pi K/4096), and R = V -
    // 2^41 K (|R| <= 2^40) is the remainder, exact in a double-float: sin(pi v)
    // keeps full relative accuracy next to the zeros of the sine.
    const ag_u64 zy = (ag_u64)x.z ^ ((ag_u64)x.w << 21);
    const ag_u64 V = zy < (1ull << 52) ? 2ull * zy + 1ull : 2ull * (zy + (zy & 1ull));
    const ag_u32 vh = (ag_u32)(V >> 32), vl = (ag_u32)V;
    const ag_u32 K = (vh + 256u) >> 9;   // (V + 2^40) >> 41
    const ag_u32 rh = vh - (K << 9);   // R = rh 2^32 + vl, rh in [-256, 255] as a signed word
    // R = Rh 2^18 + Rl with Rh = floor(R / 2^18) (|Rh| <= 2^22) and 0 <= Rl < 2^18,
    // both made exact floats by exponent tricks (no conversion unit): Rh as
    // (1.5 2^23 + Rh) - 1.5 2^23, Rl as (2^23 + Rl) - 2^23
    const int Rh = (int)((rh << 14) | (vl >> 18));
    b.fh = __int_as_float(0x4B400000 + Rh);
    b.fl = __int_as_float((int)(0x4B000000u | (vl & 0x3ffffu)));
    b.sc = ld4(kSinCosPiPeriod, (int)K);
    return b;
}
// U: the product is left unnormalised (the draw is only reassembled into a double)
template <bool U, class F>
__device__ __forceinline__ dfT<F> bm_normal(F s, dfT<F> w, F fh, F fl, dfT<F> S, dfT<F> PC) {
    const dfT<F> L = log_s<false, LOG_SRT>(s, w);
    const dfT<F> sv = sqrt_pos_(scale(L, bc<F>(-2.0f)));   // log u < 0: the argument is positive
    const dfT<F> t = fast_two_sum(fmul(fsub(fh, bc<F>(12582912.0f)), bc<F>(2.9103830456733704e-11f)),     // 2^-35
                                  fmul(fsub(fl, bc<F>(8388608.0f)), bc<F>(1.1102230246251565e-16f)));     // 2^-53
    const dfT<F> sn = sin_from_period_table(S, PC, t);
    return U ? mul_u(sv, sn) : mul(sv, sn);
}
template <bool U = false>
__device__ __forceinline__ df normal_df(ag_u64 seed, ag_u32 g, ag_u32 c) {
    const bm_words b = bm_draw(seed, g, c);
    return bm_normal<U>(b.s, b.w, b.fh, b.fl, mk(b.sc.x, b.sc.y), mk(b.sc.z, b.sc.w));
}
// The draws of two samples, g and h.
template <bool U = false>
__device__ __forceinline__ df2 normal_df(ag_u64 seed, ag_u32 g, ag_u32 h, ag_u32 c) {
    const bm_words a = bm_draw(seed, g, c), b = bm_draw(seed, h, c);
    return bm_normal<U>(pk(a.s, b.s), pair(a.w, b.w), pk(a.fh, b.fh), pk(a.fl, b.fl),
                        mk(pk(a.sc.x, b.sc.x), pk(a.sc.y, b.sc.y)), mk(pk(a.sc.z, b.sc.z), pk(a.sc.w, b.sc.w)));
}

}  // namespace e64
}  // namespace ag
