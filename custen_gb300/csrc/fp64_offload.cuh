// FP64 work moved off the FP64 pipe or to its cheapest instruction, with bit-identical results (of Divider, proved but
// for about one quotient in 2^90: see there).
//
// Sums and products as multiply-adds (F64): a multiply-add whose three operands are registers runs at 597 G/s on
// GB300, an addition or a multiplication at 503 (as does a multiply-add with a literal, parameter or zero
// operand). So a + b is fma(a, 1, b) and a b is fma(a, b, -0.0), with 1 and -0.0 in registers that the compiler
// cannot fold: the same values for all operands, signed zeros, infinities and NaN included.
//
// On GB300 one FP64 instruction of a warp holds its sub-partition's FP64 pipe for 64 cycles, while an
// integer or FP32 instruction takes one or two issue cycles. Conversions between float and double are FP64
// instructions as well (measured: 596 G conversions/s against 597 G FMA/s), a division of doubles costs 9.4
// and a reciprocal 5.6 of them. The functions below give the same bits with fewer:
//   to_double / to_float   conversions rewritten on the IEEE 754 encodings           0 instead of 1
//   div_by_float           correctly rounded c / d, d a float value                  3 instead of 10.4
//   reciprocal             correctly rounded 1 / x                                   4 instead of 5.6 (+ the range check's)
//   Divider                a / b; several a share b                                  2 + 3 per a instead of 9.4 per a
// Arguments outside the ranges named at each function take the compiler's own operation, out of line. Measured: WENO
// 1024^2 with fields of order 1, 100, 1e4, 1e6 and 1e9 (the last four with squared indicators outside div_by_float's
// range at some or all points) 226, 329, 296, 296 and 498 us, with operators throughout 412 (578 at 1e9).
//
// Method: Newton's iteration for the reciprocal (1/b = y (1 + e + e^2 + ...), e = 1 - b y), carried to about 47
// bits in pairs of floats, then one residual correction of the quotient with a fused multiply-add (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990). The
// error bounds that make the results correctly rounded stand at each function.
#pragma once

#include <cuda_runtime.h>

namespace custen {
namespace f64 {

static __device__ double g_f64_constants[2] = {1.0, -0.0};

struct F64 {
    double one, nzero;
    __device__ __forceinline__ F64() {
        const volatile double* c = g_f64_constants;
        one = c[0];
        nzero = c[1];
    }
    __device__ __forceinline__ double add(double a, double b) const { return fma(a, one, b); }
    __device__ __forceinline__ double sub(double a, double b) const { return fma(b, -one, a); }
    __device__ __forceinline__ double mul(double a, double b) const { return fma(a, b, nzero); }
};

// The compiler's own operations, for arguments outside the ranges below. Out of line: inlined, they are
// evaluated unconditionally and selected afterwards, which keeps their FP64 instructions (measured in the WENO
// kernel: 35 of 153 per point).
static __device__ __noinline__ double hw_to_double(float f) { return (double)f; }
static __device__ __noinline__ float hw_to_float(double x) { return (float)x; }
static __device__ __noinline__ double hw_multiply(double a, double b) { return a * b; }
static __device__ __noinline__ double hw_divide(double a, double b) { return a / b; }

// double of a float >= 0, times 2^scale (scale in -8 .. 0). Exact: a normal float's exponent and fraction are
// re-placed; zero stays zero. Subnormal, infinite and NaN arguments take the hardware conversion.
template <int SCALE = 0>
__device__ __forceinline__ double to_double_pos(float f) {
    const unsigned u = __float_as_uint(f);
    if (u - 0x00800000u >= 0x7f000000u && u != 0u) return hw_to_double(f) * (SCALE == 0 ? 1.0 : exp2((double)SCALE));
    const unsigned hi = u == 0u ? 0u : (u >> 3) + 0x38000000u + (unsigned)(SCALE * (1 << 20));
    return __hiloint2double((int)hi, (int)(u << 29));
}

// double of a float that is zero or normal, either sign (the caller's bounds exclude the others).
__device__ __forceinline__ double to_double_normal(float f) {
    const unsigned u = __float_as_uint(f), m = u & 0x7fffffffu;
    const unsigned hi = m == 0u ? 0u : (m >> 3) + 0x38000000u;
    return __hiloint2double((int)(hi | (u & 0x80000000u)), (int)(u << 29));
}

// Whether |x| (from its high word) is in [2^LO, 2^HI): LO, HI exponents.
template <int LO, int HI>
__device__ __forceinline__ bool exponent_in(int hi) {
    return ((unsigned)hi & 0x7fffffffu) - (unsigned)((LO + 1023) << 20) < (unsigned)((HI - LO) << 20);
}

// float of a double whose magnitude is in [2^-126, 2^128), rounded to nearest even: adding half a unit (less
// one unless the kept part is odd) below the 29 dropped bits carries into the kept ones; an overflowing carry
// gives infinity, as rounding does.
__device__ __forceinline__ float to_float_inrange(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned lo = (unsigned)b;
    const unsigned long long r = b + (0x0fffffffu + ((lo >> 29) & 1u));
    const unsigned mag = __funnelshift_l((unsigned)r, (unsigned)(r >> 32), 3) + 0x40000000u;
    return __uint_as_float((mag & 0x7fffffffu) | ((unsigned)(b >> 32) & 0x80000000u));
}

// float of a double, rounded to nearest even. Zero is handled here; magnitudes below 2^-126 or not finite in
// float take the hardware conversion.
__device__ __forceinline__ float to_float(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const bool zero = ((hi << 1) | lo) == 0u;
    if (!exponent_in<-126, 128>((int)hi) && !zero) return hw_to_float(x);
    return zero ? __uint_as_float(hi) : to_float_inrange(x);
}

// Correctly rounded c / d for a positive double c in [2^-64, 2^64) and d >= 0 a float value. d outside
// [2^-40, 2^60) takes the operator.
//   yh = RN(1/d); e = 1 - d yh is exact in float (a 24-bit by 24-bit product next to 1); yl = RN(yh (e + e^2)):
//   yh + yl is 1/d to within 2^-48 (relative). y is that sum rounded to a unit of yh's double, formed by adding
//   yl in those units to the encoding of yh; it cannot leave yh's binade downwards, since yl < 0 with yh a power
//   of two would need a float d between 2^-j and its successor. y is within 2^-47 of 1/d, q0 = RN(c y) within
//   2^-46 of c/d; the residual r = c - d q0 has at most 77 - 46 bits and is exact. q0 + r y is within 2^-93 of
//   c/d, and c/d, whose divisor has 24 bits, lies at least 2^-78 from a midpoint of two doubles: q is RN(c/d).
__device__ __forceinline__ double div_by_float(const F64& f, double c, float d) {
    const unsigned u = __float_as_uint(d);
    if (u - ((127u - 40u) << 23) >= (100u << 23)) return hw_divide(c, hw_to_double(d));
    const float yh = __frcp_rn(d);
    const float e = fmaf(-d, yh, 1.0f);
    const float yl = yh * fmaf(e, e, e);
    const unsigned uy = __float_as_uint(yh);
    // 2^(52 - exponent of yh): yl in units of the last place of yh as a double, |off| <= 2^29
    const float unit = __uint_as_float(((2u * 127u + 52u) << 23) - (uy & 0x7f800000u));
    const int off = __float2int_rn(yl * unit);
    const long long yb = ((long long)((uy >> 3) + 0x38000000u) << 32 | (long long)(uy << 29)) + off;
    const double y = __longlong_as_double(yb);
    const double dd = to_double_normal(d);
    const double q0 = f.mul(c, y);
    return fma(fma(-dd, q0, c), y, q0);
}

// 4 x for x of magnitude in [2^-1000, 2^1000), by its exponent; zero stays zero, others take the product.
__device__ __forceinline__ double times4(double x) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    const bool zero = (((unsigned)hi << 1) | (unsigned)lo) == 0u;
    if (!exponent_in<-1000, 1000>(hi) && !zero) return hw_multiply(4.0, x);
    return __hiloint2double(zero ? hi : hi + (2 << 20), lo);
}

// 1/b to within 2^-92 before its one rounding, for |b| in [2^-1000, 2^1000). An FP32 pair first, for the significand
// 1 <= s < 2 of |b|: s = bh + bl with bh the truncated float, yh = RN(1/bh), e = (1 - bh yh) - bl yh to 2^-47 (the
// parenthesis is exact), 1/s = yh + yl with yl = yh (e + e^2), renormalised so that |yl| is at most half a unit of
// yh; the sum is formed by adding yl, in units of yh's double, to yh's encoding (twice below a power of two, where
// a unit counts half), and b's exponent and sign follow there. Then one Newton step on the FP64 pipe.
__device__ __forceinline__ double reciprocal_seed(const F64& f, double b) {
    const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
    const float bh = __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x007fffffu) | 0x3f800000u);
    const float y1 = __frcp_rn(bh);
    const float bl = (float)(lo & 0x1fffffffu) * 0x1p-52f;
    const float e = __fmaf_rn(-bl, y1, __fmaf_rn(-bh, y1, 1.0f));
    const float y2 = __fmul_rn(y1, __fmaf_rn(e, e, e));
    const float yh = __fadd_rn(y1, y2);
    const float yl = __fsub_rn(y2, __fsub_rn(yh, y1));
    const unsigned uy = __float_as_uint(yh);
    const float unit = __uint_as_float(((2u * 127u + 52u) << 23) - (uy & 0x7f800000u));
    int off = __float2int_rn(yl * unit);
    if (off < 0 && (uy & 0x7fffffu) == 0u) off *= 2;
    const long long yb = ((long long)((uy >> 3) + 0x38000000u) << 32 | (long long)(uy << 29)) + off;
    const unsigned yhi = (unsigned)(yb >> 32) - ((hi & 0x7ff00000u) - 0x3ff00000u);
    const double y = __hiloint2double((int)(yhi | (hi & 0x80000000u)), (int)yb);
    return fma(y, fma(-b, y, f.one), y);
}

// Correctly rounded 1 / x. A reciprocal y within one unit in the last place becomes the correctly rounded one
// by one more iteration, except where the fraction of x is all ones (Markstein's theorem); those and arguments
// outside [2^-1000, 2^1000) take the operator.
__device__ __forceinline__ double reciprocal(const F64& f, double x) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    if (!exponent_in<-1000, 1000>(hi) || ((hi & 0xfffff) == 0xfffff && lo == -1)) return hw_divide(1.0, x);
    const double y = reciprocal_seed(f, x);
    return fma(fma(-x, y, f.one), y, y);
}

// Quotients by one divisor, correctly rounded but for the coincidence below. |b| in [2^-200, 2^200) and |a| in
// [2^-800, 2^800) or zero (the quotient and the residual's last bit, 105 places below a's first, are then normal);
// anything else takes the operator. q0 = RN(a y) is within one unit of a/b, so the residual is exact, and the
// corrected quotient is correctly rounded where y is RN(1/b) (Markstein). y is, except where 1/b lies within 2^-92
// (relative) of a midpoint, where it may be the other neighbour; q0 + r y then still differs from a/b by at most
// 2^-105 (relative), which changes a rounding only if a/b lies that near a midpoint as well. Divisors just below a
// power of two, b = 2^j (1 - k 2^-53) with small odd k, are systematically like that (1/b and quotients of simple
// numerators fall next to midpoints): fractions whose upper 20 bits are ones take the operator. For the others
// both coincidences together are about one quotient in 2^90.
struct Divider {
    double b, y;
    bool ok;
    double nzero;
    __device__ __forceinline__ Divider(const F64& f, double b_) : b(b_), nzero(f.nzero) {
        const int hi = __double2hiint(b_);
        ok = exponent_in<-200, 200>(hi) && (hi & 0xfffff) != 0xfffff;
        y = reciprocal_seed(f, b_);   // unused unless ok
    }
    __device__ __forceinline__ double operator()(double a) const {
        const unsigned hi = (unsigned)__double2hiint(a), lo = (unsigned)__double2loint(a);
        const bool zero = ((hi << 1) | lo) == 0u;
        if (!(ok && (exponent_in<-800, 800>((int)hi) || zero))) return hw_divide(a, b);
        const double q0 = fma(a, y, nzero);
        const double q = fma(fma(-b, q0, a), y, q0);
        return zero ? q0 : q;   // a zero keeps its sign
    }
};

}  // namespace f64
}  // namespace custen
