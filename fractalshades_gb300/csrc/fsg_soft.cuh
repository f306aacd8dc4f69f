// fsg_soft.cuh -- products of doubles on the integer pipes, bit for bit.
//
// An SM of GB300 issues 1.63 FP64 thread-operations a clock, 62 of 32-bit
// logic, shifts or adds and 26 of 32 x 32 + 64 -> 64-bit multiply-adds (all
// measured).  A correctly rounded 53 x 53-bit product is four of those
// multiply-adds and about a dozen others, so a loop that multiplies here and
// adds on the FP64 pipe keeps both busy: eight chains of products alone run at
// 1.6 products per SM and clock by DMUL and at 3.5 with five of the eight here.
//
// dfac is a factor: the sign and exponent fields of a double and its 53-bit
// mantissa shifted up by 6 (two 32-bit words, the upper one below 2^27, so that
// the cross products add without a carry).  dfac_mul gives the double product
// rounded to nearest even, as the multiply does, when
//   * both factors are normal with exponents within 2^+-480 (dfac_ok), so that
//     the product neither overflows nor leaves the normal range, and
//   * the 32 bits below the last kept one are not exactly 1000...0: only there
//     can the rounding depend on what lies further down (a tie, or just above
//     one).  That happens for about one product in 2^32 on mantissas without
//     structure; `ok` is cleared and the caller takes the multiply itself.
#pragma once
#include <cmath>
#include <cstring>

#include "fsg_num.cuh"

struct dfac { unsigned s, h, l; };

FSG_DEV unsigned d_hi(double x) { return (unsigned)(dbits(x) >> 32); }
FSG_DEV unsigned d_lo(double x) { return (unsigned)dbits(x); }

// normal, exponent in [-480, 479]: no product of two such leaves the normal range
#define FSG_FAC_LO (1023u - 480u)
#define FSG_FAC_N 960u
FSG_DEV bool dfac_ok(double x) { return (d_hi(x) << 1) - (FSG_FAC_LO << 21) < (FSG_FAC_N << 21); }
FSG_DEV bool dfac_ok(double2 z) { return dfac_ok(z.x) & dfac_ok(z.y); }

// the factor x 2^k (the exponent field moves: k small beside the margin of dfac_ok)
FSG_DEV dfac dfac_of(double x, int k = 0) {
    const unsigned hi = d_hi(x), lo = d_lo(x), m = (hi & 0x000fffffu) | 0x00100000u;
    dfac f;
    f.s = (hi & 0xfff00000u) + ((unsigned)k << 20);
    f.h = __funnelshift_l(lo, m, 6);
    f.l = lo << 6;
    return f;
}

// TIES: ties and what lies just above them are rounded here too (products by
// small integers, where they are common); ok is kept.  ZERO: a factor may be a
// zero of dfac_of0.
template <bool TIES, bool ZERO>
FSG_DEV double dfac_mul_t(const dfac &a, const dfac &b, bool &ok) {
    typedef unsigned long long u64;
    // the mantissas' product times 2^12, in [2^116, 2^118): v its words from 2^64 up
    const u64 t = (u64)a.l * b.l;
    u64 u = (u64)a.l * b.h + (unsigned)(t >> 32);
    u = (u64)a.h * b.l + u;
    const u64 v = (u64)a.h * b.h + (unsigned)(u >> 32);
    const unsigned vh = (unsigned)(v >> 32), vl = (unsigned)v, ul = (unsigned)u;
    const unsigned q = vh >> 21;                       // 1: the product is in [2, 4)
    const unsigned H = vh >> q, L = __funnelshift_r(vl, vh, q), r = __funnelshift_r(ul, vl, q);
    unsigned up = r >> 31;
    if (TIES) {
        const bool below = ((unsigned)t | (ul & q)) != 0u;       // bits under r
        if (r == 0x80000000u && !below) up = L & 1u;
    } else {
        ok &= r != 0x80000000u;
    }
    // exponent fields and signs add modulo 2^32 (the exponent of the result is
    // in range); H carries the mantissa's leading bit, which adds 1 to the field
    const unsigned e = a.s + b.s - 0x40000000u + (q << 20);
    u64 m = ((u64)(H + e) << 32 | L) + up;
    if (ZERO && vh == 0u) m = (u64)((a.s ^ b.s) & 0x80000000u) << 32;
    return __longlong_as_double((long long)m);
}
FSG_DEV double dfac_mul(const dfac &a, const dfac &b, bool &ok) {
    return dfac_mul_t<false, false>(a, b, ok);
}
FSG_DEV double dfac_mul_ties(const dfac &a, const dfac &b) {
    bool ok = true;
    return dfac_mul_t<true, false>(a, b, ok);
}

// The same with zero factors (derivatives that start, or stay, at zero): their
// words are 0, and the product is the zero of the factors' signs.
FSG_DEV bool dfac_ok0(double x) { return dfac_ok(x) | d_is0(x); }
FSG_DEV dfac dfac_of0(double x) {
    dfac f = dfac_of(x);
    if (d_is0(x)) { f.h = 0u; f.s = d_hi(x); }
    return f;
}
FSG_DEV double dfac_mul0(const dfac &a, const dfac &b, bool &ok) {
    return dfac_mul_t<false, true>(a, b, ok);
}

// complex products with every real product taken here and the sums on the
// FP64 pipe, in cmul's order
struct cfac { dfac x, y; };
FSG_DEV cfac cfac_of(double2 z, int k = 0) {
    cfac f;
    f.x = dfac_of(z.x, k);
    f.y = dfac_of(z.y, k);
    return f;
}
FSG_DEV double2 cfac_mul(const cfac &a, const cfac &b, bool &ok) {
    return cx(dfac_mul(a.x, b.x, ok) - dfac_mul(a.y, b.y, ok),
              dfac_mul(a.x, b.y, ok) + dfac_mul(a.y, b.x, ok));
}
// csq: the cross product on the exponent of 2 x y
FSG_DEV double2 cfac_sq(const cfac &a, bool &ok) {
    dfac x2 = a.x;
    x2.s += 0x00100000u;
    return cx(dfac_mul(a.x, a.x, ok) - dfac_mul(a.y, a.y, ok), dfac_mul(x2, a.y, ok));
}

// ---------------------------------------------------------------------------
// |z|^2 against a threshold t from upper words alone: m, the larger upper word
// of |x|, |y|, against two bounds kept 2^-15 away from where rounding matters:
//   m < lo  (|x|, |y| < sqrt(t / 2) (1 - 2^-15)): the rounded sum of the rounded
//           squares is less than t;
//   m >= hi (|x| or |y| >= sqrt(t) (1 + 2^-15)): it is greater than t -- or NaN,
//           which only an infinite or NaN part gives (m >= infinity's word).
// Between the two, a float estimate from the upper words: with sqrt(t) = f 2^E,
// f in [1/2, 1), a word less `base` and shifted is the float of |x| 2^-E with its
// mantissa cut to 20 bits (0 where it is far below), so that the sum of squares
// q has s 2^-2E in [q (1 - 2^-21), q (1 + 2^-18)]: less than t where q < tl =
// t 2^-2E (1 - 2^-17), greater where q > th = t 2^-2E (1 + 2^-20).  (A pixel whose
// derivative shrinks by 1 % a step stays 35 steps between lo and hi, and a warp
// holds 32.)
// t = 0, or a t out of 1e-290 .. 1e300, has no such bounds (for d_abs2_lt with
// t = 0, hi = 0 is one: no square is below 0).
// ---------------------------------------------------------------------------
#define FSG_INF_HI 0x7ff00000u
struct SqBound { unsigned lo, hi, base; float tl, th; };
inline unsigned fsg_hi_word(double x) {
    unsigned long long b;
    memcpy(&b, &x, 8);
    return (unsigned)(b >> 32);
}
inline SqBound fsg_sq_bound(double t) {
    SqBound b;
    b.lo = 0u;
    b.hi = FSG_INF_HI;
    b.base = 0u;
    b.tl = 0.f;
    b.th = INFINITY;
    if (!(t >= 1e-290) || !(t <= 1e300)) return b;
    b.lo = fsg_hi_word(sqrt(0.5 * t) * (1. - 0x1p-15));          // its word, rounded down
    b.hi = fsg_hi_word(sqrt(t) * (1. + 0x1p-15)) + 1u;           // and up
    int E;
    frexp(sqrt(t), &E);
    b.base = (unsigned)(E + 1023 - 127) << 20;
    const double ts = ldexp(t, -2 * E);
    b.tl = (float)(ts * (1. - 0x1p-17));
    b.th = (float)(ts * (1. + 0x1p-20));
    return b;
}
FSG_DEV unsigned d_mag_hi(double x) { return d_hi(x) & 0x7fffffffu; }
FSG_DEV unsigned d_mag_hi(double2 z) { return max(d_mag_hi(z.x), d_mag_hi(z.y)); }
// 1: |z|^2 > t, -1: |z|^2 < t, 0: open; for finite z with m in [lo, hi)
FSG_DEV int d_abs2_side(double2 z, const SqBound &b) {
    const float x = __int_as_float(max((int)(d_mag_hi(z.x) - b.base), 0) << 3);
    const float y = __int_as_float(max((int)(d_mag_hi(z.y) - b.base), 0) << 3);
    const float q = x * x + y * y;
    return q < b.tl ? -1 : q > b.th ? 1 : 0;
}
// |z|^2 > t and |z|^2 < t, t a square
FSG_DEV bool d_abs2_gt(double2 z, double t, const SqBound &b) {
    const unsigned m = d_mag_hi(z);
    if (m < b.lo) return false;
    if (m >= b.hi && m < FSG_INF_HI) return true;
    const int side = m < b.hi ? d_abs2_side(z, b) : 0;
    if (side != 0) return side > 0;
    return d_sq_gt(z.x * z.x + z.y * z.y, t);
}
FSG_DEV bool d_abs2_lt(double2 z, double t, const SqBound &b) {
    const unsigned m = d_mag_hi(z);
    if (m >= b.hi) return m >= FSG_INF_HI && d_sq_lt(z.x * z.x + z.y * z.y, t);
    if (m < b.lo) return true;
    const int side = d_abs2_side(z, b);
    if (side != 0) return side < 0;
    return d_sq_lt(z.x * z.x + z.y * z.y, t);
}
