/*
 * FP64 reciprocals, quotients, roots and comparisons on the integer pipe.
 *
 * GB300 issues one FP64 instruction per SM every 19 cycles (measured; 64 on one
 * SM sub-partition alone), and the FP64 marches keep that pipe full while the
 * integer and FP32 pipes idle (8% of the issue slots used, 14 to 25% with these), so these
 * functions form their results with integer instructions alone, half a cycle
 * each: Newton's iteration in fixed point from the FP32 hardware
 * approximation, the residual kept exactly or to 62 bits, the result rounded
 * once to 53 bits.  recip and rsq are within 0.52 ulp, in about 30 and 40
 * instructions (4 and 5 on the FP64 pipe before).  sqr_t and div_fix are the
 * IEEE root and quotient bit for bit, in about 60 and 50 (8 on the FP64 pipe
 * before; 5 from a tabulated reciprocal by Markstein's method, more without).
 * scg_divide_check, scg_root_check and scg_product_check compare them on the device.
 *
 * Operands outside the stated ranges take the division or the library
 * function behind a branch that such values alone take.
 */
#pragma once

#include <cuda_runtime.h>

namespace scg
{
namespace dev
{

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

// d's significand as an integer in [2^52, 2^53).
__device__ __forceinline__ unsigned long long sig53(unsigned hi, unsigned lo)
{
    return (static_cast<unsigned long long>((hi & 0xfffffu) | 0x100000u) << 32) | lo;
}

// 2^62 / m for the significand m in [1, 2) of d's words: with the seed
// y = Y 2^-24 the residual e = 1 - m y is exact in the low 64 bits of the
// product (|e| < 2^-21), and 1 / m = y (1 + e + e^2) up to 2^-65.  Within 2^-58
// of itself.
__device__ __forceinline__ unsigned long long rcp_sig(unsigned hi, unsigned lo)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(sig_top(hi, lo)));
    unsigned const Y = seed24(y);
    long long const E = -mul_s64_u24(static_cast<long long>(sig53(hi, lo)), Y); // e 2^76
    int const Es = static_cast<int>(E >> 24);                                   // e 2^52
    long long const T = (E >> 14) + (static_cast<long long>(Es) * Es >> 42);    // (e + e^2) 2^62
    return (static_cast<unsigned long long>(Y) << 38) +
           static_cast<unsigned long long>(mul_s64_u24((T + 4) >> 3, Y) >> 21);
}

// Reciprocal.  FP64: |d| in [2^-1022, 2^1022) as above; outside it (zero,
// subnormals, the largest magnitudes, infinities, NaN) the division.
__device__ __forceinline__ double recip(double d)
{
    unsigned const hi = static_cast<unsigned>(__double2hiint(d));
    unsigned const lo = static_cast<unsigned>(__double2loint(d));
    unsigned const e = (hi >> 20) & 0x7ffu;
    if (e - 1u > 2043u)
    {
        return 1.0 / d;
    }
    unsigned long long const bits =
        ((rcp_sig(hi, lo) + 256u) >> 9) + (static_cast<unsigned long long>(2044u - e) << 52);
    return __longlong_as_double(static_cast<long long>(bits | (static_cast<unsigned long long>(hi & 0x80000000u) << 32)));
}

// The significand's reciprocal of a divisor, for div_fix: 2^62 / m of a normal
// d, else 0 (div_fix then divides).
__device__ __forceinline__ unsigned long long rcp_fix(double d)
{
    unsigned const hi = static_cast<unsigned>(__double2hiint(d));
    unsigned const e = (hi >> 20) & 0x7ffu;
    return e - 1u < 2046u ? rcp_sig(hi, static_cast<unsigned>(__double2loint(d))) : 0ull;
}

static __device__ __noinline__ double div_plain(double x, double d) { return x / d; }
// Calls, not instructions that the compiler could predicate: a predicated
// multiplication takes its turn in the FP64 pipe whether or not it is wanted.
static __device__ __noinline__ double mul_native(double a, double b) { return __dmul_rn(a, b); }
static __device__ __noinline__ double mul_plain(double a, double b)
{
    unsigned const ha = static_cast<unsigned>(__double2hiint(a)), hb = static_cast<unsigned>(__double2hiint(b));
    bool const za = ((ha << 1) | static_cast<unsigned>(__double2loint(a))) == 0u;
    bool const zb = ((hb << 1) | static_cast<unsigned>(__double2loint(b))) == 0u;
    if ((za && (hb & 0x7fffffffu) < 0x7ff00000u) || (zb && (ha & 0x7fffffffu) < 0x7ff00000u))
    {
        return __hiloint2double(static_cast<int>((ha ^ hb) & 0x80000000u), 0);
    }
    return mul_native(a, b);
}

// x / d rounded to nearest, from r = rcp_fix(d): bit for bit the IEEE quotient.
// For a normal x whose quotient is normal, Z is the significands' quotient
// within 0.53 units (of its 53 bits) and its exact remainder, modulo 2^64, says
// whether it is one off; a quotient is never half-way between two.  A zero x
// gives a zero; anything else divides.
__device__ __forceinline__ double div_fix(double x, double d, unsigned long long r)
{
    unsigned const hx = static_cast<unsigned>(__double2hiint(x)), lx = static_cast<unsigned>(__double2loint(x));
    unsigned const hd = static_cast<unsigned>(__double2hiint(d)), ld = static_cast<unsigned>(__double2loint(d));
    unsigned const ex = (hx >> 20) & 0x7ffu;
    unsigned const e = ex - ((hd >> 20) & 0x7ffu) + 1023u; // of a quotient of significands >= 1
    unsigned long long const sign = static_cast<unsigned long long>((hx ^ hd) & 0x80000000u) << 32;
    if (r == 0ull || ex - 1u > 2045u || e - 2u > 2043u)
    {
        bool const zero = r != 0ull && ((hx << 1) | lx) == 0u;
        return zero ? __longlong_as_double(static_cast<long long>(sign)) : div_plain(x, d);
    }
    unsigned long long const ma = sig53(hx, lx), mb = sig53(hd, ld);
    unsigned const low = ma >= mb ? 0u : 1u;
    unsigned const sh = 9u - low;
    unsigned long long Z = (mul_hi64(ma << 11, r) + (256ull >> low)) >> sh; // (ma / mb) 2^(52 + low)
    long long const rem2 = 2 * static_cast<long long>((ma << (52u + low)) - Z * mb);
    long long const b = static_cast<long long>(mb);
    Z += static_cast<unsigned long long>((rem2 > b ? 1 : 0) - (rem2 < -b ? 1 : 0));
    return __longlong_as_double(
        static_cast<long long>((Z + (static_cast<unsigned long long>(e - 1u - low) << 52)) | sign));
}

// a * b rounded to nearest even: bit for bit the FP64 product, from the exact
// 128-bit product of the significands in integers (about 36 instructions and
// four wide multiplications, 18 SM cycles beside the FP64 pipe's 19), for
// marches that fill the FP64 pipe.  For normal operands with a normal product;
// others (zeros among them) take a call that only they make.
__device__ __forceinline__ double mul_int(double a, double b)
{
    unsigned const ha = static_cast<unsigned>(__double2hiint(a)), la = static_cast<unsigned>(__double2loint(a));
    unsigned const hb = static_cast<unsigned>(__double2hiint(b)), lb = static_cast<unsigned>(__double2loint(b));
    unsigned const ea = (ha >> 20) & 0x7ffu, eb = (hb >> 20) & 0x7ffu;
    unsigned const e = ea + eb - 1023u; // of a product of significands below 2
    if (ea - 1u > 2045u || eb - 1u > 2045u || e - 1u > 2044u)
    {
        return mul_plain(a, b);
    }
    // A = m_a 2^63 and B = m_b 2^55, significands m in [1, 2): the product's high
    // word is m_a m_b 2^54, the low word only says whether it is exact.
    unsigned long long const A = sig53(ha, la) << 11, B = sig53(hb, lb) << 3;
    unsigned const ah = static_cast<unsigned>(A >> 32), al = static_cast<unsigned>(A);
    unsigned const bh = static_cast<unsigned>(B >> 32), bl = static_cast<unsigned>(B);
    unsigned long long const p0 = static_cast<unsigned long long>(al) * bl;
    unsigned long long const p1 = static_cast<unsigned long long>(al) * bh + (p0 >> 32);
    unsigned long long const p2 = static_cast<unsigned long long>(ah) * bl + static_cast<unsigned>(p1);
    unsigned long long P = static_cast<unsigned long long>(ah) * bh + (p1 >> 32) + (p2 >> 32);
    P |= (static_cast<unsigned>(p0) | static_cast<unsigned>(p2)) != 0u ? 1ull : 0ull;
    unsigned const big = static_cast<unsigned>(P >> 55); // product of significands >= 2
    unsigned const sh = 2u + big;
    unsigned long long const m = (P + ((P >> sh) & 1ull) + (1u + 2u * big)) >> sh; // in [2^52, 2^53]
    return __longlong_as_double(static_cast<long long>(
        (m + (static_cast<unsigned long long>(e - 1u + big) << 52)) |
        (static_cast<unsigned long long>((ha ^ hb) & 0x80000000u) << 32)));
}

// Whether x is a positive normal number.
__device__ __forceinline__ bool pos_normal(unsigned hi) { return hi - 0x00100000u < 0x7fe00000u; }

// Reciprocal root of m in [1, 4), the significand of a positive normal x
// taken with its exponent's parity: x = m 4^h.  X = m 2^62; returns
// 2^62 / sqrt(m).  With the seed y, e = 1 - m y^2 to 2^-61 (|e| < 2^-20) and
// 1 / sqrt(m) = y (1 + e / 2 + 3 e^2 / 8) up to 2^-61.
__device__ __forceinline__ unsigned long long rsq_core(float top, unsigned long long X, unsigned odd)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(__float_as_uint(top) + (odd << 23))));
    unsigned const Y = seed24(y);
    unsigned long long const Z = static_cast<unsigned long long>(Y) * Y << 16; // y^2 2^64
    long long const E = static_cast<long long>((1ull << 62) - mul_hi64(X, Z)); // e 2^62
    int const Es = static_cast<int>(E >> 12);                                   // e 2^50
    unsigned const sq = static_cast<unsigned>(static_cast<unsigned long long>(static_cast<long long>(Es) * Es) >> 32);
    long long const T = E + static_cast<long long>(sq * 3u >> 8); // (e + 3 e^2 / 4) 2^62
    return (static_cast<unsigned long long>(Y) << 38) +
           static_cast<unsigned long long>(mul_s64_u24((T + 4) >> 3, Y) >> 22);
}
__device__ __forceinline__ unsigned long long rsq_fixed(unsigned hi, unsigned lo, unsigned long long & X, int & h)
{
    int const k = static_cast<int>(hi >> 20) - 1023;
    h = k >> 1;
    unsigned const odd = static_cast<unsigned>(k) & 1u;
    X = sig53(hi, lo) << (10u + odd);
    return rsq_core(sig_top(hi, lo), X, odd);
}

// 1 / |g|, |g|^2 = tiny + sum g_d^2 with tiny = 1e-200, as w 2^(-62 - h) from the
// exact squares' upper 61 bits at the largest component's scale (14 instructions
// a component), where no component reaches 2^500; false for others.  For ND FP64
// instructions of an element's and an equation's: a substep of 2M triangles
// 1331 -> 1252 us, 384k tetrahedra 688 -> 659, 64k hexahedra 298 -> 285.
template <int ND>
__device__ __forceinline__ bool inverse_norm(double const * g, unsigned long long & w, int & h)
{
    constexpr unsigned FLOOR = 690; // exponent of 2^-333: its square against tiny
    constexpr unsigned long long TINY = static_cast<unsigned long long>(1e-200 * 0x1p400 * 0x1p325);
    unsigned e[ND], top = FLOOR;
#pragma unroll
    for (int d = 0; d < ND; ++d)
    {
        e[d] = (static_cast<unsigned>(__double2hiint(g[d])) >> 20) & 0x7ffu;
        top = max(top, e[d]);
    }
    // (g / 2^(top - 1023))^2 2^59, each below 2^61.
    unsigned long long q = TINY >> min(2u * (top - FLOOR), 63u);
#pragma unroll
    for (int d = 0; d < ND; ++d)
    {
        unsigned long long const m = sig53(static_cast<unsigned>(__double2hiint(g[d])),
                                           static_cast<unsigned>(__double2loint(g[d])))
                                     << 11;
        q += mul_hi64(m, m) >> min(2u * (top - e[d]) + 3u, 63u);
    }
    unsigned const lz = static_cast<unsigned>(__clzll(static_cast<long long>(q)));
    int const k = 2 * (static_cast<int>(top) - 1023) + 4 - static_cast<int>(lz);
    unsigned const odd = static_cast<unsigned>(k) & 1u;
    q <<= lz;
    h = k >> 1;
    w = rsq_core(__uint_as_float((127u << 23) | (static_cast<unsigned>(q >> 40) & 0x7fffffu)), q >> (1u - odd), odd);
    return top < 1523u;
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

// sqrt(x): FP64 positive normal x rounded to nearest, as the library's root is,
// and zero; else, and in FP32, the library's.  With x / sqrt(x) rounded to S, in
// units of its 53 bits within 0.52 of the root, the exact remainder of S^2,
// modulo 2^64, says whether S is one off: a root is never half-way between two.
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
    unsigned long long S = (mul_hi64(X, r) + 128u) >> 8; // sqrt(m) 2^52
    long long const rem = static_cast<long long>((X << 42) - S * S);
    long long const s = static_cast<long long>(S);
    S += static_cast<unsigned long long>((rem > s ? 1 : 0) - (rem <= -s ? 1 : 0));
    return __longlong_as_double(
        static_cast<long long>(S + (static_cast<unsigned long long>(1022 + h) << 52)));
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
