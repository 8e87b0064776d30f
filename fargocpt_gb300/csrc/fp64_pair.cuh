// FP64-accurate arithmetic from pairs of FP32 values for the FP64 form's
// kernels: a value is the unevaluated sum hi + lo of two floats with |lo|
// at most about ulp(hi) / 2, about 48 significant bits.  GB300 issues FP32
// operations at about 70 times its FP64 rate (measured: 113 against 1.6
// results per clock per SM), so a pair operation of 5 to 20 FP32 operations
// is several times cheaper than one FP64 operation.
//
// The building blocks are the error-free transformations TwoSum (Knuth 1969),
// Fast2Sum (Dekker 1971) and TwoProduct by fused multiply-add, combined as in
// Joldes, Muller and Popescu, "Tight and rigorous error bounds for basic
// building blocks of double-word arithmetic" (ACM TOMS 44, 2017): the sum of
// two pairs (their algorithm 6, relative error below 3 u^2, u = 2^-24) and the
// product of two pairs (algorithm 12, below 5 u^2).  Every operation is spelled
// with the round-to-nearest intrinsics so that the compiler neither contracts nor
// reorders them.
#pragma once

#include <cuda_runtime.h>

namespace fgpu {

struct f2 {
    float h, l;
};

// a + b exactly as s + e, for |a| >= |b| or a = 0
__device__ __forceinline__ f2 fast_two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b);
    return f2{s, __fsub_rn(b, __fsub_rn(s, a))};
}
// a + b exactly as s + e, any magnitudes
__device__ __forceinline__ f2 two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    return f2{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
// a b exactly as p + e
__device__ __forceinline__ f2 two_prod(float a, float b)
{
    const float p = __fmul_rn(a, b);
    return f2{p, __fmaf_rn(a, b, -p)};
}

__device__ __forceinline__ f2 f2_add(f2 x, f2 y)
{
    const f2 s = two_sum(x.h, y.h);
    const f2 t = two_sum(x.l, y.l);
    const f2 v = fast_two_sum(s.h, __fadd_rn(s.l, t.h));
    return fast_two_sum(v.h, __fadd_rn(t.l, v.l));
}
__device__ __forceinline__ f2 f2_neg(f2 x) { return f2{-x.h, -x.l}; }
__device__ __forceinline__ f2 f2_sub(f2 x, f2 y) { return f2_add(x, f2_neg(y)); }

__device__ __forceinline__ f2 f2_mul(f2 x, f2 y)
{
    const f2 c = two_prod(x.h, y.h);
    const float t = __fmaf_rn(x.h, y.l, __fmul_rn(x.l, y.l));
    return fast_two_sum(c.h, __fadd_rn(c.l, __fmaf_rn(x.l, y.h, t)));
}
// 1 / sqrt(d) for d > 0: the hardware estimate, one FP32 Newton step, then
// one Newton step whose residual 1 - d r^2 is formed in pair arithmetic; the
// result is within a few units of 2^-46 of the exact value
__device__ __forceinline__ f2 f2_rsqrt(f2 d)
{
    float r = rsqrtf(d.h);
    r = __fmul_rn(r, __fmaf_rn(__fmul_rn(-0.5f, d.h), __fmul_rn(r, r), 1.5f));
    const f2 p = f2_mul(d, two_prod(r, r));  // about 1
    const float e = __fsub_rn(__fsub_rn(1.0f, p.h), p.l);
    return fast_two_sum(r, __fmul_rn(__fmul_rn(0.5f, r), e));
}

// running sum hi + lo of pairs, one TwoSum per term (the low parts are small
// against the sum, their float addition loses only below 2^-48 of it)
__device__ __forceinline__ void f2_accumulate(float &hi, float &lo, f2 x)
{
    const f2 s = two_sum(hi, x.h);
    hi = s.h;
    lo = __fadd_rn(lo, __fadd_rn(s.l, x.l));
}

// ---------------------------------------------------------------------------
// Conversions on the integer pipe.  GB300 converts between FP64 and FP32
// (F2F) at about one result per clock per SM, slower than its FP64
// arithmetic, so the transports split doubles into pairs and join pairs into
// doubles with bit operations and one integer-to-float conversion.
// ---------------------------------------------------------------------------

// x as a pair, |x - (h + l)| <= 2^-48 |x|, |l| < ulp(h): h is x truncated to
// 24 significant bits (the sign, the rebased exponent and the top 23
// mantissa bits, shifted into place), l the remaining 29 mantissa bits
// converted to float and scaled by 2^(e - 1075).  (The pair is not
// renormalised: the pair operations take |l| < ulp(h) with error bounds at
// most twice those for |l| <= ulp(h) / 2, and the sign of h is the sign of
// x.)  Both are normal floats for biased exponents e in [949, 1150]
// (2^-74 <= |x| < 2^128).  Below that range x becomes zero (an absolute
// error under 2^-74); at or above it, and for infinities and NaN, a NaN of
// x's sign, so that a state out of the pairs' range shows as non-finite.
// Branch-free: the callers' loops over a thread's cells stay one
// instruction stream.
__device__ __forceinline__ f2 f2_split(double x)
{
    const unsigned w1 = (unsigned)__double2hiint(x), w0 = (unsigned)__double2loint(x);
    const unsigned ax = w1 & 0x7fffffffu, sign = w1 & 0x80000000u;
    const unsigned hb = __funnelshift_l(w0, ax - (896u << 20), 3);
    const float scale = __uint_as_float((hb & 0x7f800000u) - (52u << 23));
    const unsigned lb = __float_as_uint(__fmul_rn(__uint2float_rn(w0 & 0x1fffffffu), scale));
    const bool in = ax - (949u << 20) < (202u << 20);
    const unsigned out = ax < (949u << 20) ? 0u : (0x7fc00000u | sign);
    return f2{__uint_as_float(in ? (hb | sign) : out), __uint_as_float(in ? (lb | sign) : out)};
}

// h + l as a double, rounded to nearest even as the FP64 addition of the two
// would be, on the integer pipe: h's bits are the double's top (24 significant
// bits, exact), and l, scaled to the double's units 2^(e - 1075) and rounded
// to an integer by F2I, is added to the bit pattern as one 64-bit integer (the
// patterns of a binade and its neighbours are consecutive, so a carry into the
// exponent is the right value).  A low part of the other sign than h's can
// step into the binade below when h is a power of two; its units are then that
// binade's, hence the exponent of h's bit pattern less one.  Zero and subnormal
// h give zero, infinities and NaN a NaN.  Branch-free.
// The FP64 addition it replaces runs at 1.6 results per clock per SM; this
// runs at 3.7 (measured back to back, split and rounding included).
__device__ __forceinline__ double f2_to_double(f2 a)
{
    const unsigned b = __float_as_uint(a.h);
    const unsigned mag = b & 0x7fffffffu, sign = b & 0x80000000u;
    const unsigned lr = __float_as_uint(a.l) ^ sign;  // l relative to h's sign
    // 2^(52 - exponent) as a float; below 2^-75 the scale stays at its largest
    const unsigned e = max((mag - (lr >> 31)) & 0x7f800000u, 52u << 23);
    const int li = __float2int_rn(__fmul_rn(__uint_as_float(lr), __uint_as_float((306u << 23) - e)));
    const unsigned long long v =
        (((unsigned long long)((mag >> 3) + (896u << 20)) << 32) | (b << 29)) + (long long)li;
    const bool normal = mag - 0x00800000u < 0x7f000000u;
    const unsigned out = mag < 0x00800000u ? 0u : (sign | 0x7ff80000u);
    return __hiloint2double((int)(normal ? (unsigned)(v >> 32) | sign : out),
                            (int)(normal ? (unsigned)v : 0u));
}

// ---------------------------------------------------------------------------
// Cheaper pair operations for the transports, whose error bars are relative
// to the operands' magnitudes (the pair representation itself carries 2^-48
// of each value): the sloppy sum (Joldes, Muller and Popescu, algorithm 5),
// absolute error within a few 2^-48 (|x| + |y|); the product without the
// low-by-low term; the quotient from the hardware reciprocal
// estimate (rcp.approx, within 2^-22) with one correction in pair
// arithmetic, relative error within a few 2^-46.
// ---------------------------------------------------------------------------
__device__ __forceinline__ f2 f2_sadd(f2 x, f2 y)
{
    const f2 s = two_sum(x.h, y.h);
    return fast_two_sum(s.h, __fadd_rn(s.l, __fadd_rn(x.l, y.l)));
}
__device__ __forceinline__ f2 f2_ssub(f2 x, f2 y) { return f2_sadd(x, f2_neg(y)); }

__device__ __forceinline__ f2 f2_smul(f2 x, f2 y)
{
    const f2 c = two_prod(x.h, y.h);
    return fast_two_sum(c.h, __fadd_rn(c.l, __fmaf_rn(x.l, y.h, __fmul_rn(x.h, y.l))));
}
// x + a d in one: the product's error-free high part, the sum's TwoSum, one
// renormalisation
__device__ __forceinline__ f2 f2_sfma(f2 x, f2 a, f2 d)
{
    const f2 p = two_prod(a.h, d.h);
    const float pl = __fmaf_rn(a.l, d.h, __fmaf_rn(a.h, d.l, p.l));
    const f2 s = two_sum(x.h, p.h);
    return fast_two_sum(s.h, __fadd_rn(s.l, __fadd_rn(x.l, pl)));
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float rsqrt_approx(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// sqrt(x) for x > 0: x rsqrt(x)
__device__ __forceinline__ f2 f2_sqrt(f2 x) { return f2_smul(x, f2_rsqrt(x)); }

// p / s for a normal s: q = p.h rcp(s.h), then q + (p - q s) rcp(s.h)
__device__ __forceinline__ f2 f2_sdiv(f2 p, f2 s)
{
    const float r = rcp_approx(s.h);
    const float q = __fmul_rn(p.h, r);
    // p.h - q s.h in one rounding (q s.h is within a few ulps of p.h)
    const float d = __fmaf_rn(-q, s.l, __fadd_rn(__fmaf_rn(-q, s.h, p.h), p.l));
    return fast_two_sum(q, __fmul_rn(d, r));
}

// ---------------------------------------------------------------------------
// Two pairs at a time: every operation is the packed FP32 instruction of the
// two values (add, mul, fma .rn.f32x2), which rounds each as the scalar one
// does, so a packed operation gives the bits of the scalar functions above.
// GB300's FP32 pipe takes a packed instruction for two cycles (measured: 120
// results per clock per SM packed, 119 scalar), so packing does not speed the
// arithmetic itself; it halves the issue slots it takes, which the loads,
// selects and integer conversions around it need.
// ---------------------------------------------------------------------------
struct f2x2 {
    float2 h, l;
};

__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 vneg(float2 a) { return make_float2(-a.x, -a.y); }
// a - b (the product by -1 is exact)
__device__ __forceinline__ float2 vsub(float2 a, float2 b)
{
    return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}
__device__ __forceinline__ float2 vrcp(float2 a)
{
    return make_float2(rcp_approx(a.x), rcp_approx(a.y));
}

__device__ __forceinline__ f2x2 pack(f2 a, f2 b)
{
    return f2x2{make_float2(a.h, b.h), make_float2(a.l, b.l)};
}
__device__ __forceinline__ f2x2 pack(f2 a) { return pack(a, a); }
__device__ __forceinline__ f2 first(f2x2 a) { return f2{a.h.x, a.l.x}; }
__device__ __forceinline__ f2 second(f2x2 a) { return f2{a.h.y, a.l.y}; }

__device__ __forceinline__ f2x2 fast_two_sum(float2 a, float2 b)
{
    const float2 s = vadd(a, b);
    return f2x2{s, vsub(b, vsub(s, a))};
}
__device__ __forceinline__ f2x2 two_sum(float2 a, float2 b)
{
    const float2 s = vadd(a, b);
    const float2 bb = vsub(s, a);
    return f2x2{s, vadd(vsub(a, vsub(s, bb)), vsub(b, bb))};
}
__device__ __forceinline__ f2x2 two_prod(float2 a, float2 b)
{
    const float2 p = vmul(a, b);
    return f2x2{p, vfma(a, b, vneg(p))};
}
__device__ __forceinline__ f2x2 f2_neg(f2x2 x) { return f2x2{vneg(x.h), vneg(x.l)}; }
__device__ __forceinline__ f2x2 f2_sadd(f2x2 x, f2x2 y)
{
    const f2x2 s = two_sum(x.h, y.h);
    return fast_two_sum(s.h, vadd(s.l, vadd(x.l, y.l)));
}
__device__ __forceinline__ f2x2 f2_ssub(f2x2 x, f2x2 y)
{
    // two_sum of x.h and -y.h with the signs carried by the subtractions
    const float2 s = vsub(x.h, y.h);
    const float2 bb = vsub(s, x.h);
    const float2 e = vsub(vsub(x.h, vsub(s, bb)), vadd(y.h, bb));
    return fast_two_sum(s, vadd(e, vsub(x.l, y.l)));
}
__device__ __forceinline__ f2x2 f2_smul(f2x2 x, f2x2 y)
{
    const f2x2 c = two_prod(x.h, y.h);
    return fast_two_sum(c.h, vadd(c.l, vfma(x.l, y.h, vmul(x.h, y.l))));
}
__device__ __forceinline__ f2x2 f2_sfma(f2x2 x, f2x2 a, f2x2 d)
{
    const f2x2 p = two_prod(a.h, d.h);
    const float2 pl = vfma(a.l, d.h, vfma(a.h, d.l, p.l));
    const f2x2 s = two_sum(x.h, p.h);
    return fast_two_sum(s.h, vadd(s.l, vadd(x.l, pl)));
}
// 1 / sqrt(d) for d > 0: the hardware estimate, one FP32 Newton step, then
// one whose residual 1 - d r^2 is formed from the error-free square of r
__device__ __forceinline__ f2x2 f2_rsqrt(f2x2 d)
{
    float2 r = make_float2(rsqrtf(d.h.x), rsqrtf(d.h.y));
    const float2 half = make_float2(0.5f, 0.5f), one = make_float2(1.f, 1.f);
    const float2 mh = vneg(d.h);
    r = vmul(r, vfma(vmul(half, mh), vmul(r, r), make_float2(1.5f, 1.5f)));
    const f2x2 r2 = two_prod(r, r);
    const float2 e = vfma(vneg(d.l), r2.h, vfma(mh, r2.l, vfma(mh, r2.h, one)));
    return fast_two_sum(r, vmul(vmul(half, r), e));
}
__device__ __forceinline__ f2x2 f2_sdiv(f2x2 p, f2x2 s)
{
    const float2 r = vrcp(s.h);
    const float2 q = vmul(p.h, r);
    const float2 nq = vneg(q);
    const float2 d = vfma(nq, s.l, vadd(vfma(nq, s.h, p.h), p.l));
    return fast_two_sum(q, vmul(d, r));
}

}  // namespace fgpu
