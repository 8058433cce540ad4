// IEEE double arithmetic on the integer pipe, for the FP64 sweeps.
//
// On this part one FP64 instruction of any kind (add, multiply, FMA, compare,
// float<->double conversion) occupies its SM quadrant's FP64 unit for 64
// cycles whatever the number of active lanes and however independent the
// instructions are (probe, one warp: 64.6 cycles at 1 and at 4 independent
// chains; four warps on four quadrants: 64-77 each), while an integer add
// costs 1.2 and a shift, logic operation or 32 x 32 -> 64 multiply 2.2
// cycles.  A correctly rounded product in integers is about 25 instructions,
// ~45 cycles once its operands are unpacked, and runs beside the FP64 unit,
// which is left to the additions.  Everything here returns the bits of the
// IEEE operation (round to nearest, ties to even) for the operands it
// accepts, and says when it does not accept them, so the sweeps keep the bits
// of the FP64 instructions.
//
// The same code compiles for the host and is checked there against the host's
// IEEE arithmetic (tests/test_int64.py).
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef __CUDACC__
#ifndef VA_HD
#define VA_HD
#endif
#else
#ifndef VA_HD
#define VA_HD __host__ __device__
#endif
#endif

namespace va {

VA_HD inline uint64_t f64_bits(double v)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t u;
    std::memcpy(&u, &v, 8);
    return u;
#endif
}
VA_HD inline double f64_from_bits(uint64_t u)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double v;
    std::memcpy(&v, &u, 8);
    return v;
#endif
}
VA_HD inline uint32_t f64_hi(double v) { return (uint32_t)(f64_bits(v) >> 32); }
VA_HD inline uint32_t f64_lo(double v) { return (uint32_t)f64_bits(v); }

VA_HD inline uint64_t umulhi64(uint64_t a, uint64_t b)
{
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
VA_HD inline int64_t smulhi64(int64_t a, int64_t b)
{
#ifdef __CUDA_ARCH__
    return __mul64hi(a, b);
#else
    return (int64_t)(((__int128)a * b) >> 64);
#endif
}

// ------------------------------------------------------------- comparisons

constexpr uint64_t kF64Inf = 0x7ff0000000000000ull;

// v != v
VA_HD inline bool is_nan64(double v) { return (f64_bits(v) & ~(1ull << 63)) > kF64Inf; }
// |v| < inf
VA_HD inline bool is_finite64(double v) { return (f64_hi(v) & 0x7ff00000u) != 0x7ff00000u; }
// v > c for a constant c > 0 and any v (false for a NaN)
VA_HD inline bool greater_pos64(double v, double c)
{
    const uint64_t cb = f64_bits(c);
    return f64_bits(v) - cb - 1 < kF64Inf - cb;
}
// v <= c for a constant c > 0 and any v (false for a NaN)
VA_HD inline bool less_equal_pos64(double v, double c)
{
    return !greater_pos64(v, c) && !is_nan64(v);
}
// 0 < v < inf
VA_HD inline bool positive_finite64(double v) { return f64_bits(v) - 1 < kF64Inf - 1; }
// a > b for numbers >= +0, neither of them a NaN
VA_HD inline bool greater_nonneg64(double a, double b) { return f64_bits(a) > f64_bits(b); }
// the larger of two numbers >= +0, neither of them a NaN
VA_HD inline double max_nonneg64(double a, double b) { return f64_bits(a) > f64_bits(b) ? a : b; }

// ---------------------------------------------------------------- products
//
// Operands are unpacked once and used in several products: the first factor
// as its 53-bit significand shifted to the top of 64 bits, the second as its
// significand times two, so the product of two non-zero operands lies in
// [2^116, 2^118) and its upper 64 bits hold the 53 or 54 leading bits.  The
// low 64 bits, reduced to 32 with a sticky bit, decide the rounding through
// the carry of (low + half - 1 + lsb).  Sign and exponent fields are added as
// they stand; the significand's hidden bit and its possible carry to 2^53
// ride on the same addition.

struct MulL { // first factor
    uint32_t h, l, e;
};
struct MulR { // second factor
    uint32_t h, l, e;
};

// Range of the operands seen so far: `beyond(e)` when one of them was neither
// zero nor within 2^-e .. 2^(e+1) in magnitude, e <= 960 (infinities, NaNs
// and subnormals included).
struct MulRange {
    uint32_t mn = 0xffffffffu, mx = 0;
    VA_HD void note(uint32_t hi, uint32_t lo)
    {
        const uint32_t u = hi + hi; // the sign is shifted out
        // a zero becomes the largest value here, a subnormal below 2^-1042 stays 0
        const uint32_t v = u - (lo == 0 ? 1u : 0u);
        mn = v < mn ? v : mn;
        mx = u > mx ? u : mx;
    }
    VA_HD bool beyond(int e) const { return mn < (uint32_t)(1023 - e) << 21 || mx >= (uint32_t)(1024 + e) << 21; }
};

// _in: an operand known to be in range (a constant, a product of noted values)
VA_HD inline MulL mul_left_in(double a)
{
    const uint32_t hi = f64_hi(a), lo = f64_lo(a), u = hi + hi;
    const uint32_t m = (hi & 0xfffffu) | (u < 0x100000u ? u : 0x100000u); // hidden bit, none for a zero
    return {(m << 11) | (lo >> 21), lo << 11, hi & 0xfff00000u};
}
VA_HD inline MulR mul_right_in(double b)
{
    const uint32_t hi = f64_hi(b), lo = f64_lo(b), u = hi + hi;
    const uint32_t m = (hi & 0xfffffu) | (u < 0x100000u ? u : 0x100000u);
    return {(m << 1) | (lo >> 31), lo << 1, hi & 0xfff00000u};
}
VA_HD inline MulL mul_left(double a, MulRange &r)
{
    r.note(f64_hi(a), f64_lo(a));
    return mul_left_in(a);
}
VA_HD inline MulR mul_right(double b, MulRange &r)
{
    r.note(f64_hi(b), f64_lo(b));
    return mul_right_in(b);
}
// -a, and -2 a for an operand in range
VA_HD inline MulL mul_neg(MulL a) { return {a.h, a.l, a.e ^ 0x80000000u}; }
VA_HD inline MulL mul_m2(MulL a) { return {a.h, a.l, (a.e + 0x100000u) ^ 0x80000000u}; }

// The correctly rounded product of two unpacked operands (in range).
VA_HD inline double mul_rn(MulL a, MulR b)
{
    const uint64_t p00 = (uint64_t)a.l * b.l, p01 = (uint64_t)a.l * b.h;
    const uint64_t p10 = (uint64_t)a.h * b.l, p11 = (uint64_t)a.h * b.h;
    const uint64_t mid = p01 + (p00 >> 32);                        // < 2^55
    const uint64_t low = (mid & 0xffffffffu) + (p10 & 0xffffffffu); // bits 32..63 and a carry
    const uint64_t top = p11 + (mid >> 32) + (p10 >> 32) + (low >> 32);
    const uint32_t th = (uint32_t)(top >> 32), tl = (uint32_t)top;
    const uint32_t f0 = (uint32_t)p00;
    const uint32_t frac = (uint32_t)low | (f0 < 1u ? f0 : 1u); // low half, sticky in bit 0
    const uint32_t s = th >> 21;                               // product >= 2^117
    // (th : tl : frac) >> s, the sticky bit kept
    const uint32_t mh = th >> s;
#ifdef __CUDA_ARCH__
    const uint32_t ml = __funnelshift_r(tl, th, s);
    const uint32_t fr = __funnelshift_r(frac, tl, s) | (frac & 1u);
#else
    const uint32_t ml = s ? (tl >> 1) | (th << 31) : tl;
    const uint32_t fr = (s ? (frac >> 1) | (tl << 31) : frac) | (frac & 1u);
#endif
    const uint64_t round = (uint64_t)fr + 0x7fffffffu + (ml & 1u); // carries when the fraction rounds up
    const uint64_t lo = (uint64_t)ml + (round >> 32);
    const uint32_t ex = a.e + b.e + (s << 20) - 0x40000000u; // less the bias and the hidden bit
    const uint32_t hi = mh + ex + (uint32_t)(lo >> 32);
    const uint32_t h = th ? hi : (a.e ^ b.e) & 0x80000000u; // a zero factor
    return f64_from_bits(((uint64_t)h << 32) | (uint32_t)lo);
}


// --------------------------------------------------------------- quotients
//
// n / d correctly rounded for positive normal n, d with a normal quotient
// (false otherwise): three digits of 21 bits from a float reciprocal, each
// with its exact remainder.  The digits leave |remainder| <= 2.5 d at 2^-63,
// so the quotient is known to 2.5 units of 2^-63; only where that straddles a
// rounding boundary (10 or 11 bits below the last place) is the remainder
// reduced exactly.  A quotient of two doubles is never halfway between two.
VA_HD inline bool div_rn_pos(double n, double d, double &q)
{
    const uint64_t nb = f64_bits(n), db = f64_bits(d);
    const int en = (int)(nb >> 52), ed = (int)(db >> 52);
    // normal operands (a sign bit fails too) and a quotient well inside the range
    if ((unsigned)(en - 1) >= 2046u || (unsigned)(ed - 1) >= 2046u || (unsigned)(en - ed + 1000) >= 2000u)
        return false;
    const uint64_t N = (nb & 0xfffffffffffffull) | (1ull << 52), D = (db & 0xfffffffffffffull) | (1ull << 52);
    const float df = (float)(int32_t)(D >> 29);
#ifdef __CUDA_ARCH__
    const float y = __fdividef(2097152.0f, df);
#else
    const float y = 2097152.0f / df;
#endif
    const int64_t q1 = (int64_t)(int32_t)rintf((float)(int32_t)(N >> 29) * y);
    const int64_t r1 = (int64_t)(N << 21) - q1 * (int64_t)D;
    const int64_t q2 = (int64_t)(int32_t)rintf((float)(int32_t)(r1 >> 29) * y);
    const int64_t r2 = (int64_t)((uint64_t)r1 << 21) - q2 * (int64_t)D;
    const int64_t q3 = (int64_t)(int32_t)rintf((float)(int32_t)(r2 >> 29) * y);
    int64_t r3 = (int64_t)((uint64_t)r2 << 21) - q3 * (int64_t)D;
    uint64_t Q = ((uint64_t)q1 << 42) + (uint64_t)(q2 * (1 << 21)) + (uint64_t)q3; // n / d = (Q + r3 / D) 2^-63
    const int big = (int)(Q >> 63);                                                // n / d >= 1
    const uint32_t half = 512u << big;
    uint32_t frac = (uint32_t)Q & (2 * half - 1);
    bool up = frac > half;
    if (frac - half + 4 <= 8) { // within the digits' error of the boundary
        while (r3 < 0) {
            r3 += (int64_t)D;
            Q--;
        }
        while (r3 >= (int64_t)D) {
            r3 -= (int64_t)D;
            Q++;
        }
        // the boundary is Q' = (.. half): above it, or on it with a remainder
        frac = (uint32_t)Q & (2 * half - 1);
        up = frac >= half;
    }
    const uint64_t m = (Q >> (10 + big)) + (up ? 1 : 0);
    q = f64_from_bits(((uint64_t)(en - ed + 1021 + big) << 52) + m);
    return true;
}

// n / d for n >= 0, d > 0 or any NaN: the integer form, else the FP64 division
// (a zero, subnormal or infinite operand or quotient)
VA_HD inline double quotient64(double n, double d)
{
    double q;
    if (!div_rn_pos(n, d, q))
        q = n / d;
    return q;
}

} // namespace va
