/*
 * FP64 divisions and roots that cost fewer FP64-pipe instructions than the
 * IEEE operations.
 *
 * div_rcp: division by a tabulated reciprocal, rounded exactly as x / d.
 *
 * A march that divides many times by grid-only quantities (widths,
 * spacings) can store r = 1 / d once, rounded to nearest, and recover the
 * correctly rounded quotient from it with Markstein's method (P. Markstein,
 * "Computation of elementary functions on the IBM RISC System/6000
 * processor", IBM J. Res. Dev. 34(1), 1990; the theorem is also stated in
 * Muller et al., "Handbook of Floating-Point Arithmetic"):
 *
 *   q0 = x r                  within 1.5 ulp of x / d (r within half an ulp)
 *   q1 = q0 + (x - q0 d) r    within one ulp (the correction's own error is
 *                             about 2^-53 of q0's)
 *   q2 = q1 + (x - q1 d) r    = x / d rounded to nearest (Markstein's
 *                             theorem: r within half an ulp of 1 / d, q1
 *                             within one ulp, the remainder x - q1 d exact
 *                             in a fused multiply-add)
 *
 * one multiplication and four fused multiply-adds, all on values of the
 * march.  The theorem needs the operands away from the ends of the exponent
 * range (no overflow or underflow in q, the remainder or the correction), so
 * both |x| and |d| must lie in [2^-400, 2^400); a zero x is exact too (q0
 * carries its sign, which the corrections would lose).  Anything else
 * (denormals, infinities, NaN, a d whose reciprocal was not tabulated)
 * divides.  The results equal CUDA's IEEE division bit for bit; the device
 * check scg_divide_check compares the two.
 *
 * recip, rsq, sqr_t: reciprocals and roots within 0.52 ulp, on the integer
 * pipe (below).
 */
#pragma once

#include <cuda_runtime.h>

namespace scg
{
namespace dev
{

// High word of |v| against [2^-400, 2^400): biased exponents 623 to 1422.
constexpr unsigned RCP_EXP_LO = (1023u - 400u) << 20;
constexpr unsigned RCP_EXP_SPAN = 800u << 20;

__device__ __forceinline__ bool rcp_window(double v)
{
    unsigned const h = static_cast<unsigned>(__double2hiint(v)) & 0x7fffffffu;
    return h - RCP_EXP_LO < RCP_EXP_SPAN;
}

// The tabulated reciprocal of d: 1 / d rounded to nearest when d is in the
// window, else 0 (div_rcp then divides).
__device__ __forceinline__ double rcp_tab(double d) { return rcp_window(d) ? 1.0 / d : 0.0; }

static __device__ __noinline__ double div_plain(double x, double d) { return x / d; }

// x / d, rounded to nearest, from r = rcp_tab(d).
__device__ __forceinline__ double div_rcp(double x, double d, double r)
{
    double const q0 = x * r;
    unsigned const hx = static_cast<unsigned>(__double2hiint(x)) & 0x7fffffffu;
    bool const xok = hx - RCP_EXP_LO < RCP_EXP_SPAN || (hx | static_cast<unsigned>(__double2loint(x))) == 0u;
    if (__double2hiint(r) != 0 && xok)
    {
        double const q1 = __fma_rn(__fma_rn(-q0, d, x), r, q0);
        double const q2 = __fma_rn(__fma_rn(-q1, d, x), r, q1);
        return copysign(q2, q0);
    }
    return div_plain(x, d);
}

// ---------------------------------------------------------------------------
// Reciprocals and roots on the integer pipe.
//
// GB300 issues one FP64 instruction per SM every 16 cycles, and the FP64
// marches keep that pipe ~88% busy while the integer and FP32 pipes idle (8%
// of the issue slots used), so these functions form their results with
// integer instructions alone: Newton's iteration in fixed point from the FP32
// hardware approximation, the residual kept exactly or to 62 bits, the result
// rounded once to 53 bits.  About 30 (recip), 40 (rsq) and 48 (sqr) integer
// instructions in place of 4, 5 and 8 of the FP64 pipe (a triangle's substep
// takes 6, 12 and 2 of them, a hexahedron's 15, 40 and 2).
// Results are within 0.52 ulp (scg_divide_check and scg_root_check compare
// them on the device).
//
// Operands outside the stated ranges take the division or the library
// function behind a branch that such values alone take.

// |d|'s top 24 significand bits as a float in [1, 2).
__device__ __forceinline__ float sig_top(unsigned hi, unsigned lo)
{
    return __uint_as_float((127u << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29));
}

// A seed y in (0.5, 1] as a 24-bit integer y 2^24, kept inside [2^23, 2^24).
__device__ __forceinline__ unsigned seed24(float y)
{
    unsigned const b = min(max(__float_as_uint(y), 0x3f000000u), 0x3f7fffffu);
    return (b & 0x7fffffu) | 0x800000u;
}

// t * y for a signed 64-bit t and y below 2^24, modulo 2^64.
__device__ __forceinline__ long long mul_s64_u24(long long t, unsigned y)
{
    unsigned long long const u = static_cast<unsigned long long>(t);
    unsigned long long const lo = static_cast<unsigned long long>(static_cast<unsigned>(u)) * y;
    return static_cast<long long>(lo + (static_cast<unsigned long long>(static_cast<unsigned>(u >> 32) * y) << 32));
}

// a * b / 2^64 up to two units of the result.
__device__ __forceinline__ unsigned long long mul_hi64(unsigned long long a, unsigned long long b)
{
    unsigned const ah = static_cast<unsigned>(a >> 32), al = static_cast<unsigned>(a);
    unsigned const bh = static_cast<unsigned>(b >> 32), bl = static_cast<unsigned>(b);
    return static_cast<unsigned long long>(ah) * bh + __umulhi(ah, bl) + __umulhi(al, bh);
}

// Reciprocal.  FP64, |d| in [2^-1022, 2^1022): with m = |d|'s significand
// (m 2^52 an integer) and the seed y = Y 2^-24, the residual e = 1 - m y is
// exact in the low 64 bits of the product (|e| < 2^-21), and
// 1 / m = y (1 + e + e^2) up to 2^-65.  Outside that range (zero, subnormals,
// the largest magnitudes, infinities, NaN) the division.  FP32: the division.
__device__ __forceinline__ double recip(double d)
{
    unsigned const hi = static_cast<unsigned>(__double2hiint(d));
    unsigned const lo = static_cast<unsigned>(__double2loint(d));
    unsigned const e = (hi >> 20) & 0x7ffu;
    if (e - 1u > 2043u)
    {
        return 1.0 / d;
    }
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(sig_top(hi, lo)));
    unsigned const Y = seed24(y);
    unsigned long long const m =
        (static_cast<unsigned long long>((hi & 0xfffffu) | 0x100000u) << 32) | lo;
    long long const E = -mul_s64_u24(static_cast<long long>(m), Y); // e 2^76
    int const Es = static_cast<int>(E >> 24);                       // e 2^52
    long long const T = (E >> 14) + (static_cast<long long>(Es) * Es >> 42); // (e + e^2) 2^62
    unsigned long long const r = (static_cast<unsigned long long>(Y) << 38) +
                                 static_cast<unsigned long long>(mul_s64_u24((T + 4) >> 3, Y) >> 21); // 2^62 / m
    unsigned long long const bits = ((r + 256u) >> 9) + (static_cast<unsigned long long>(2044u - e) << 52);
    return __longlong_as_double(static_cast<long long>(bits | (static_cast<unsigned long long>(hi & 0x80000000u) << 32)));
}
__device__ __forceinline__ float recip(float d) { return 1.0f / d; }

// Whether x is a positive normal number.
__device__ __forceinline__ bool pos_normal(unsigned hi) { return hi - 0x00100000u < 0x7fe00000u; }

// Reciprocal root of m in [1, 4), the significand of a positive normal x
// taken with its exponent's parity: x = m 4^h.  X = m 2^62; returns
// 2^62 / sqrt(m).  With the seed y, e = 1 - m y^2 to 2^-61 (|e| < 2^-20) and
// 1 / sqrt(m) = y (1 + e / 2 + 3 e^2 / 8) up to 2^-61.
__device__ __forceinline__ unsigned long long rsq_fixed(unsigned hi, unsigned lo, unsigned long long & X, int & h)
{
    int const k = static_cast<int>(hi >> 20) - 1023;
    h = k >> 1;
    unsigned const odd = static_cast<unsigned>(k) & 1u;
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(__float_as_uint(sig_top(hi, lo)) + (odd << 23))));
    unsigned const Y = seed24(y);
    X = ((static_cast<unsigned long long>((hi & 0xfffffu) | 0x100000u) << 32) | lo) << (10u + odd);
    unsigned long long const Z = static_cast<unsigned long long>(Y) * Y << 16; // y^2 2^64
    long long const E = static_cast<long long>((1ull << 62) - mul_hi64(X, Z)); // e 2^62
    int const Es = static_cast<int>(E >> 12);                                   // e 2^50
    unsigned const sq = static_cast<unsigned>(static_cast<unsigned long long>(static_cast<long long>(Es) * Es) >> 32);
    long long const T = E + static_cast<long long>(sq * 3u >> 8); // (e + 3 e^2 / 4) 2^62
    return (static_cast<unsigned long long>(Y) << 38) +
           static_cast<unsigned long long>(mul_s64_u24((T + 4) >> 3, Y) >> 22);
}

// 1 / sqrt(x): FP64 positive normal x as above, else the library's; FP32 the
// library's.
__device__ __forceinline__ double rsq(double x)
{
    unsigned const hi = static_cast<unsigned>(__double2hiint(x));
    if (!pos_normal(hi))
    {
        return rsqrt(x);
    }
    unsigned long long X;
    int h;
    unsigned long long const r = rsq_fixed(hi, static_cast<unsigned>(__double2loint(x)), X, h);
    return __longlong_as_double(
        static_cast<long long>(((r + 256u) >> 9) + (static_cast<unsigned long long>(1021 - h) << 52)));
}
__device__ __forceinline__ float rsq(float x) { return rsqrtf(x); }

// sqrt(x) = x / sqrt(x): FP64 positive normal x and zero, else the library's;
// FP32 the library's.
__device__ __forceinline__ double sqr_t(double x)
{
    unsigned const hi = static_cast<unsigned>(__double2hiint(x));
    unsigned const lo = static_cast<unsigned>(__double2loint(x));
    if (!pos_normal(hi))
    {
        return ((hi << 1) | lo) == 0u ? x : sqrt(x);
    }
    unsigned long long X;
    int h;
    unsigned long long const r = rsq_fixed(hi, lo, X, h);
    unsigned long long const q = mul_hi64(X, r); // sqrt(m) 2^60
    return __longlong_as_double(
        static_cast<long long>(((q + 128u) >> 8) + (static_cast<unsigned long long>(1022 + h) << 52)));
}
__device__ __forceinline__ float sqr_t(float x) { return sqrtf(x); }

// Comparisons of FP64 values on the integer pipe (a DSETP issues on the FP64
// pipe): the bit patterns of non-negative values order as signed integers,
// and every negative value's is below them.
__device__ __forceinline__ bool lt_nonneg(double a, double b) // a < b for a >= 0
{
    return __double_as_longlong(a) < __double_as_longlong(b);
}
__device__ __forceinline__ double max_pos(double m, double u) // the larger of u and m >= +0
{
    return lt_nonneg(m, u) ? u : m;
}
__device__ __forceinline__ double min_neg(double m, double u) // the smaller of u and m <= -0
{
    return static_cast<unsigned long long>(__double_as_longlong(m)) <
                   static_cast<unsigned long long>(__double_as_longlong(u))
               ? u
               : m;
}

} // namespace dev
} // namespace scg
