// gbh_df.cuh -- double-float arithmetic on FP32 instructions, and exact
// float <-> double conversions on the integer pipe.
//
// A df value is an unevaluated sum hi + lo of two floats with |lo| <=
// ulp(hi)/2, carrying about 48 significand bits. The primitives are the
// error-free transformations of Dekker (1971) and Knuth (TAOCP vol. 2,
// 4.2.2): TwoSum, FastTwoSum and TwoProd via fused multiply-add, composed as
// in the double-double literature (Hida, Li, Bailey 2001, "sloppy" add).
//
// On GB300 the FP64 pipe takes one warp instruction (an addition as much as a
// multiply-add) per 19 clocks of an SM, 1.7 lanes a clock, while FP32 runs
// ~113 FFMA lanes, and the F2F conversions between float and double cost as
// much as two DFMAs, so the mixed-precision step keeps gate and table
// arithmetic in df and converts with integer bit manipulation instead of F2F.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gbh {

struct df {
    float hi, lo;
};

__device__ __forceinline__ df df_make(float h, float l) { df r; r.hi = h; r.lo = l; return r; }

__device__ __forceinline__ df two_sum(float a, float b)
{
    const float s = a + b;
    const float bb = s - a;
    const float e = (a - (s - bb)) + (b - bb);
    return df_make(s, e);
}

__device__ __forceinline__ df fast_two_sum(float a, float b)
{
    const float s = a + b;
    return df_make(s, b - (s - a));
}

__device__ __forceinline__ df two_prod(float a, float b)
{
    const float p = a * b;
    return df_make(p, __fmaf_rn(a, b, -p));
}

__device__ __forceinline__ df df_add(df x, df y)
{
    df s = two_sum(x.hi, y.hi);
    s.lo += x.lo + y.lo;
    return fast_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ df df_add_f(df x, float y)
{
    df s = two_sum(x.hi, y);
    s.lo += x.lo;
    return fast_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ df df_neg(df x) { return df_make(-x.hi, -x.lo); }

__device__ __forceinline__ df df_mul(df x, df y)
{
    df p = two_prod(x.hi, y.hi);
    p.lo = __fmaf_rn(x.hi, y.lo, p.lo);
    p.lo = __fmaf_rn(x.lo, y.hi, p.lo);
    return fast_two_sum(p.hi, p.lo);
}

__device__ __forceinline__ df df_mul_f(df x, float y)
{
    df p = two_prod(x.hi, y);
    p.lo = __fmaf_rn(x.lo, y, p.lo);
    return fast_two_sum(p.hi, p.lo);
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// x / y: one float quotient, its df remainder, one correction
__device__ __forceinline__ df df_div(df x, df y)
{
    const float r = rcp_approx(y.hi);
    const float q1 = x.hi * r;
    df p = two_prod(q1, y.hi);
    p.lo = __fmaf_rn(q1, y.lo, p.lo);
    const float rem = ((x.hi - p.hi) - p.lo) + x.lo;
    const float q2 = rem * r;
    return fast_two_sum(q1, q2);
}

// ---- exact conversions on the integer pipe --------------------------------
// double -> float truncated toward zero (exact when the double already has at
// most 24 significant bits; values below the float normal range flush to 0)
__device__ __forceinline__ float d2f_trunc_bits(double d)
{
    const uint32_t hi = (uint32_t)__double2hiint(d);
    const uint32_t lo = (uint32_t)__double2loint(d);
    const uint32_t sign = hi & 0x80000000u;
    const int e = (int)((hi >> 20) & 0x7ffu) - 896;
    const uint32_t m = ((hi & 0xfffffu) << 3) | (lo >> 29);
    const uint32_t bits = (e <= 0) ? sign : (e >= 255 ? (sign | 0x7f800000u) : (sign | ((uint32_t)e << 23) | m));
    return __uint_as_float(bits);
}

// double -> df on the integer pipe: hi = d truncated to 24 significant bits,
// lo = the next 24 bits of the significand, truncated (|d - hi - lo| <
// 2^-47 |d|); no FP64 instruction. Values whose hi or lo falls outside the
// float normal range lose that part (flush to signed zero).
__device__ __forceinline__ df d2df(double d)
{
    const uint32_t h = (uint32_t)__double2hiint(d);
    const uint32_t l = (uint32_t)__double2loint(d);
    const float fh = d2f_trunc_bits(d);
    const uint32_t r = l & 0x1fffffffu;
    const int e = (int)((h >> 20) & 0x7ffu);
    const int p = 31 - __clz((int)r);
    const int fe = p + e - 948;
    uint32_t lo = 0u;
    if (r != 0u && fe > 0 && e - 896 > 0 && e - 896 < 255) {
        const uint32_t m = p >= 23 ? (r >> (p - 23)) : (r << (23 - p));
        lo = (h & 0x80000000u) | ((uint32_t)fe << 23) | (m & 0x7fffffu);
    }
    return df_make(fh, __uint_as_float(lo));
}

// The same for a voltage: |d| is taken into [2^-126, 2^128), so that a zero
// costs 1e-38 V and a NaN or infinity shows as a voltage beyond 1e38 V; the
// low 29 bits through one integer-to-float conversion, truncated as d2df
// truncates them (rounded, they moved the trace of a neuron at its threshold
// by 4e-8). A third fewer instructions than d2df.
__device__ __forceinline__ df d2df_volt(double d)
{
    const uint32_t h = (uint32_t)__double2hiint(d), l = (uint32_t)__double2loint(d);
    const uint32_t a = min(max(h & 0x7fffffffu, 0x38100000u), 0x47efffffu), sign = h & 0x80000000u;
    const uint32_t hi = __funnelshift_l(l, a - 0x38000000u, 3) | sign;
    const uint32_t unit = (uint32_t)max((int)(a >> 20) - 948, 0) << 23 | sign;   // the last place of d
    return df_make(__uint_as_float(hi), __uint2float_rz(l & 0x1fffffffu) * __uint_as_float(unit));
}

// df -> double on the integer pipe: lo's significand, shifted to hi's unit in
// the last place and rounded there to nearest even, is added to or taken from
// hi's bits: the FP64 sum of the two (hi below the float normal range gives a
// signed zero). No FP64 instruction: the FP64 unit takes one warp instruction
// per 19 clocks of an SM, an addition as much as a multiply-add. Needs |lo|
// below hi's unit in the last place (any df but an unfinished one).
__device__ __forceinline__ double df2d(df x)
{
    const uint32_t uh = __float_as_uint(x.hi), ul = __float_as_uint(x.lo);
    const uint32_t eh = (uh >> 23) & 0xffu, el = (ul >> 23) & 0xffu;
    const uint32_t sign = uh & 0x80000000u;
    const uint32_t h = ((uh & 0x7fffffffu) >> 3) + 0x38000000u, l = uh << 29;
    const bool minus = (int)(uh ^ ul) < 0;
    // lo in units of 2^-52 of hi's binade, half of that where the difference
    // falls below hi's power of two: its 24 bits, 7 places up and sh down
    const uint32_t sh = eh - max(el, 1u) - 22u - (minus && (uh & 0x7fffffu) == 0u ? 1u : 0u);
    const uint32_t a = ((ul & 0x7fffffu) | (el ? 0x800000u : 0u)) << 7;
    const uint32_t m = sh < 32u ? (a + (1u << (sh - 1u)) - 1u + ((a >> sh) & 1u)) >> sh : 0u;
    const uint64_t mag = ((uint64_t)h << 32) | l;
    const uint64_t r = minus ? mag - m : mag + m;
    return __hiloint2double(eh == 0u ? (int)sign : (int)((uint32_t)(r >> 32) | sign), eh == 0u ? 0 : (int)(uint32_t)r);
}

// df -> double for values whose error of 2^-126 does not matter (a row's
// right-hand side in volts, its diagonal above 1): exact conversions that
// take a zero for 2^-127, one FP64 addition; half the instructions of df2d.
__device__ __forceinline__ double f2d_raw(float f)
{
    const uint32_t u = __float_as_uint(f);
    return __hiloint2double((int)((((u & 0x7fffffffu) >> 3) + 0x38000000u) | (u & 0x80000000u)), (int)(u << 29));
}
__device__ __forceinline__ double df2d_row(df x) { return f2d_raw(x.hi) + f2d_raw(x.lo); }

// Reciprocal of a normal double to about 2^-44, the seed of the FP64 corrections
// below: one Newton step without FP64 instructions, the significand m in [1,2)
// as a float pair, a float seed r (MUFU), its residual e = 1 - m r on FP32
// multiply-adds (below 2^-22, so it and r e are off by 2^-46), and r + r e
// assembled on the integer pipe, r e in units of 2^-53. Valid for
// 2^-1021 < |b| < 2^1021.
__device__ __forceinline__ double rcp_seed(double b)
{
    const uint32_t hi = (uint32_t)__double2hiint(b), lo = (uint32_t)__double2loint(b);
    const float mh = __uint_as_float(0x3f800000u | (__funnelshift_l(lo, hi, 3) & 0x7fffffu));
    const float ml = (float)(lo & 0x1fffffffu) * 0x1p-52f;
    const float r = rcp_approx(mh);
    const float e = __fmaf_rn(-ml, r, __fmaf_rn(-mh, r, 1.0f));
    const int c = __float2int_rn(r * e * 0x1p53f);
    const uint32_t ru = __float_as_uint(r);
    const uint64_t y = (((uint64_t)((ru >> 3) + 0x38000000u) << 32) | (ru << 29)) + (uint64_t)(int64_t)c;
    const uint32_t yh = ((uint32_t)(y >> 32) + 0x3ff00000u - (hi & 0x7ff00000u)) | (hi & 0x80000000u);
    return __hiloint2double((int)yh, (int)(uint32_t)y);
}

// The mixed form's reciprocal: one Newton step r + r e in FP64's own precision,
// fma(r, fma(-b, r, 1), r) to its last place, without an FP64 instruction. The
// residual e = 1 - m r of the significand m (53 bits) and the seed r (24 bits)
// is formed exactly in 76 fraction bits modulo 1 (it is below 2^-21) and
// rounded at 2^-53, where the product r e is rounded to r's last place. With
// e in FP32 pairs the reciprocal was good to 2^-43.8 instead of this step's
// 2^-44 (100,000 cables of 16: 27.9 us a step, 28.3 so, 28.9 with all of e's
// bits in the product).
__device__ __forceinline__ double rcp_step(double b)
{
    const uint32_t hi = (uint32_t)__double2hiint(b), lo = (uint32_t)__double2loint(b);
    const float r = rcp_approx(__uint_as_float(0x3f800000u | (__funnelshift_l(lo, hi, 3) & 0x7fffffu)));
    const uint32_t ru = __float_as_uint(r), R = ru - 0x3e800000u;   // r in [1/2, 1], times 2^24
    const uint64_t p = (uint64_t)R * lo + (1u << 22);
    const uint32_t ph = (uint32_t)(p >> 32) + R * ((hi & 0xfffffu) | 0x100000u);
    const int32_t e = (int32_t)__funnelshift_r((uint32_t)p, ph, 23);   // -e times 2^53, rounded
    const int32_t c = (int32_t)(((int64_t)(int32_t)R * e + (1 << 23)) >> 24);
    const uint64_t y = (((uint64_t)((ru >> 3) + 0x38000000u) << 32) | (ru << 29)) - (uint64_t)(int64_t)c;
    const uint32_t yh = ((uint32_t)(y >> 32) + 0x3ff00000u - (hi & 0x7ff00000u)) | (hi & 0x80000000u);
    return __hiloint2double((int)yh, (int)(uint32_t)y);
}

// Are the exponents of all operands within 2^+-450? Quotients, reciprocals
// and the residuals of the corrections below are then normal numbers.
__device__ __forceinline__ bool mid_range(double a)
{
    return ((uint32_t)__double2hiint(a) & 0x7ff00000u) - ((1023u - 450u) << 20) <= (900u << 20);
}

// May b be divided by through rcp_seed: mid_range, and its first 20 fraction
// bits not all ones. Just below a power of two, 1 / b lies next to the middle
// between two doubles (1 / (2 - k 2^-52) = 1/2 + k 2^-54 + k^2 2^-107 ...),
// closer than the seed's Newton step can tell.
__device__ __forceinline__ bool divisor_ok(double b)
{
    return mid_range(b) && ((uint32_t)__double2hiint(b) & 0xfffffu) != 0xfffffu;
}

// IEEE division, out of line: operands the corrected quotients do not cover
// (zeros, infinities, NaN, far exponents, divisors just below a power of two).
__device__ __noinline__ static double div_ieee(double a, double b) { return a / b; }

// 1 / b, correctly rounded: one Newton step y + y (1 - b y) in two FMAs from a
// seed good to 2^-44. Before its rounding the step is off by 2^-88, so the
// result is the correctly rounded one unless 1/b lies within 2^-88 of the
// middle between two doubles (of the other divisors one in 2^34; there it may
// be the neighbour: for quotients through div_by, see rcp_exact). 2 FP64
// instructions against the division's 5.5.
__device__ __forceinline__ double rcp_rn(double b)
{
    if (!divisor_ok(b)) return div_ieee(1.0, b);
    const double y = rcp_seed(b);
    return fma(y, fma(-b, y, 1.0), y);
}

// RN(1 / b) without exception, for a reciprocal that is a result of its own:
// the step once more. From the result or its neighbour e = 1 - b z is exact and
// below 2^-53, so before its rounding the step is off by e^2 < 2^-106 of it;
// and 1/b is 2^-106 of itself or more from the middle between two doubles (b's
// 53 bits times the middle's 54 differ from 2^106). 4 FP64 instructions.
__device__ __forceinline__ double rcp_exact(double b)
{
    if (!divisor_ok(b)) return div_ieee(1.0, b);
    const double y = rcp_seed(b), z = fma(y, fma(-b, y, 1.0), y);
    return fma(z, fma(-b, z, 1.0), z);
}

// RN(a / b) from y = rcp_rn(b) by Markstein's correction (P. Markstein, IBM
// Journal of Research and Development 34, 1990): q = RN(a y) is within an ulp
// of a / b, its residual a - b q is exact in one FMA, and RN(q + residual y)
// is the correctly rounded quotient for a correctly rounded y. (Where y is
// its neighbour the correction is off by 2^-52 ulp of q, which shows only if
// a / b is that close to the middle between two doubles besides.) Needs a
// and b in mid_range.
__device__ __forceinline__ double div_by(double a, double b, double y)
{
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}

// RN(a / b): 5 FP64 instructions against the division's 9.
__device__ __forceinline__ double div_rn(double a, double b)
{
    if (!(mid_range(a) && divisor_ok(b))) return div_ieee(a, b);
    const double y = rcp_seed(b);
    return div_by(a, b, fma(y, fma(-b, y, 1.0), y));
}

}  // namespace gbh
