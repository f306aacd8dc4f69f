// fsg_soft.cuh -- products of doubles on the integer pipes, bit for bit.
//
// An SM of GB300 issues 1.6 FP64 thread-operations a clock, 61 of 32-bit
// logic or shifts and 26 of 32 x 32 + 64 -> 64-bit multiply-adds (measured on
// eight independent chains a thread, 4 CTAs of 256 an SM: 0.503e12, 19.1e12 and
// 8.2e12 a second at 2070 MHz).  A correctly rounded 53 x 53-bit product is four of those
// multiply-adds and about a dozen others, so a loop that multiplies here and
// adds on the FP64 pipe keeps both busy: eight chains of products alone run at
// 1.6 products per SM and clock by DMUL, at 4.2 with five of the eight here and at
// 3.0 with all of them here (0.503, 1.32 and 0.95e12 a second).
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

// a + b and a * b where the code asks for them and nowhere ahead of their branch
FSG_DEV double d_mul_here(double a, double b) {
#ifdef __CUDA_ARCH__
    double r;
    asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
    return r;
#else
    return a * b;
#endif
}
FSG_DEV double d_add_here(double a, double b) {
#ifdef __CUDA_ARCH__
    double r;
    asm volatile("add.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
    return r;
#else
    return a + b;
#endif
}
FSG_DEV unsigned d_hi(double x) { return (unsigned)(dbits(x) >> 32); }
FSG_DEV unsigned d_lo(double x) { return (unsigned)dbits(x); }

// x with its sign bit xored by s (0 or 0x80000000): the product by 1 or -1
FSG_DEV double d_flip(double x, unsigned s) {
    return __hiloint2double((int)(d_hi(x) ^ s), (int)d_lo(x));
}

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
    // the rounding bit, at the top of r; a tie to the even neighbour
    unsigned top = r;
    if (TIES) {
        const bool below = ((unsigned)t | (ul & q)) != 0u;       // bits under r
        if (r == 0x80000000u && !below) top = L << 31;
    } else {
        ok &= r != 0x80000000u;
    }
    // exponent fields and signs add modulo 2^32 (the exponent of the result is
    // in range); H carries the mantissa's leading bit, which adds 1 to the field
    const unsigned e = a.s + b.s - 0x40000000u + (q << 20);
    unsigned lo, hi;
#ifdef __CUDA_ARCH__
    // (the top bit as the carry of top + top)
    asm("{ .reg .u32 c; add.cc.u32 c, %2, %2; addc.cc.u32 %0, %3, 0; addc.u32 %1, %4, %5; }"
        : "=r"(lo), "=r"(hi) : "r"(top), "r"(L), "r"(H), "r"(e));
#else
    const u64 m = ((u64)(H + e) << 32 | L) + (top >> 31);
    lo = (unsigned)m;
    hi = (unsigned)(m >> 32);
#endif
    if (ZERO && vh == 0u) { lo = 0u; hi = (a.s ^ b.s) & 0x80000000u; }
    return __hiloint2double((int)hi, (int)lo);
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
// the same with zero parts allowed in a (its factors from dfac_of0)
FSG_DEV cfac cfac_of0(double2 z) {
    cfac f;
    f.x = dfac_of0(z.x);
    f.y = dfac_of0(z.y);
    return f;
}
FSG_DEV double2 cfac_mul0(const cfac &a, const cfac &b, bool &ok) {
    return cx(dfac_mul0(a.x, b.x, ok) - dfac_mul0(a.y, b.y, ok),
              dfac_mul0(a.x, b.y, ok) + dfac_mul0(a.y, b.x, ok));
}
// csq: the cross product on the exponent of 2 x y
FSG_DEV double2 cfac_sq(const cfac &a, bool &ok) {
    dfac x2 = a.x;
    x2.s += 0x00100000u;
    return cx(dfac_mul(a.x, a.x, ok) - dfac_mul(a.y, a.y, ok), dfac_mul(x2, a.y, ok));
}

// Whether the four products of a and b are normal, for parts of any normal size
// (dfac_ok instead bounds each part).  Without `zeros` a zero part refuses; with
// it, zero parts of a are left aside (dfac_of0).
template <bool ZEROS>
FSG_DEV bool cfac_ok(double2 a, double2 b) {
    unsigned ax = d_hi(a.x) & 0x7ff00000u, ay = d_hi(a.y) & 0x7ff00000u;
    const unsigned bx = d_hi(b.x) & 0x7ff00000u, by = d_hi(b.y) & 0x7ff00000u;
    if (ZEROS) {
        if (d_is0(a.x)) ax = ay;
        if (d_is0(a.y)) ay = ax;
    }
    const unsigned la = min(ax, ay), ha = max(ax, ay), lb = min(bx, by), hb = max(bx, by);
    return (min(la, lb) != 0u) & (max(ha, hb) != 0x7ff00000u) & (la + lb >= 1025u << 20)
           & (ha + hb <= 3068u << 20);
}

// ---------------------------------------------------------------------------
// A factor of any size, for loops whose values range from 1 to far below
// 2^-480: its exponent field f tells products that are normal from those that
// round to zero (a zero factor, or a product below 2^-1075) and from the rest
// (subnormal results, overflow, infinities and NaN), which clear ok.
// ---------------------------------------------------------------------------
struct sfac { unsigned s, h, l; int f; };
#define FSG_F_ZERO (-10000)
#define FSG_F_SUB 5000
#define FSG_F_INF 20000
FSG_DEV sfac sfac_of(double x, int k = 0) {
    const dfac d = dfac_of(x, k);
    const int e = (int)(d_hi(x) >> 20 & 0x7ffu);
    sfac f;
    f.s = d.s; f.h = d.h; f.l = d.l;
    f.f = e == 0x7ff ? FSG_F_INF : e == 0 ? (d_is0(x) ? FSG_F_ZERO : FSG_F_SUB) : e + k;
    return f;
}
FSG_DEV double sfac_mul(const sfac &a, const sfac &b, bool &ok) {
    dfac p, q;
    p.s = a.s; p.h = a.h; p.l = a.l;
    q.s = b.s; q.h = b.h; q.l = b.l;
    bool kept = true;
    const double m = dfac_mul(p, q, kept);
    const int e = a.f + b.f;
    const bool zero = e <= 968;                 // below 2^(968 - 2044) = 2^-1076
    ok &= zero | (kept & (unsigned)(e - 1025) <= 3068u - 1025u);
    return zero ? d_zero(((a.s ^ b.s) >> 31) != 0u) : m;
}

// cmul, by the integer products where they can be (out of line elsewhere)
static __device__ __noinline__ double2 cmul_full(double2 a, double2 b) { return cmul(a, b); }
FSG_DEV double2 cmul_soft(double2 a, double2 b) {
    bool ok = dfac_ok(a) & dfac_ok(b);
    double2 r = cfac_mul(cfac_of(a), cfac_of(b), ok);
    if (!ok) r = cmul_full(a, b);
    return r;
}

// ---------------------------------------------------------------------------
// Values m 2^e (xc): sums of two on one frame.  A sum of doubles rounds the same
// on any power of two, so the value of p 2^ep + q 2^eq does not depend on the
// frame it is taken on, while nothing leaves the normal range: the bits are
// those of the reference's co-exponent sum.
// ---------------------------------------------------------------------------
FSG_DEV int d_field(double x) { return (int)(d_hi(x) >> 20 & 0x7ffu); }      // biased exponent
// x 2^d for a normal x whose result is normal, 0 for 0
FSG_DEV double d_shift(double x, int d) {
    const int hi = (int)d_hi(x) + (d_is0(x) ? 0 : d << 20);
    return __hiloint2double(hi, (int)d_lo(x));
}
// r = p 2^ep + q 2^eq, part by part.  A part 55 or more binary orders below the
// other's leaves it as it is; where that holds for both parts there is no sum to
// take.  ok is cleared where q does not fit p's frame.
FSG_DEV xc frame_add(double2 p, int ep, double2 q, int eq, bool &ok) {
    const int d = eq - ep;
    const int px = d_field(p.x), py = d_field(p.y), qx = d_field(q.x), qy = d_field(q.y);
    const int gx = px - qx - d, gy = py - qy - d;
    if (min(gx, gy) >= 55 && min(px, py) > 0) return xc_make(p.x, p.y, ep);
    if (max(gx, gy) <= -55 && min(qx, qy) > 0) return xc_make(q.x, q.y, eq);
    ok &= ((unsigned)(qx + d - 1) < 2045u) | d_is0(q.x);
    ok &= ((unsigned)(qy + d - 1) < 2045u) | d_is0(q.y);
    return xc_make(p.x + d_shift(q.x, d), p.y + d_shift(q.y, d), ep);
}
// a + b, with a sum only where one takes part in the other: 56 binary orders
// apart (or beside a zero or a subnormal) the larger is the sum; two zeros add to
// -0 where both are
FSG_DEV double d_add_far(double a, double b) {
    const int g = d_field(a) - d_field(b);
    if (g >= 56) return a;
    if (g <= -56) return b;
    if (d_is0(a) & d_is0(b)) return d_zero(((d_hi(a) & d_hi(b)) >> 31) != 0u);
    return d_add_here(a, b);
}
// the larger part's exponent field (0 for zero and subnormal parts)
FSG_DEV int d_field_max(double2 z) { return max(d_field(z.x), d_field(z.y)); }
FSG_DEV int d_field_min(double2 z) { return min(d_field(z.x), d_field(z.y)); }
// back to a frame with the larger part in 2^+-100 (one shift for both parts);
// ok is cleared where the smaller part would leave the normal range
FSG_DEV void frame_renorm(xc &a, bool &ok) {
    const int k = d_field_max(xm(a)) - 1023;
    if ((unsigned)(k + 100) <= 200u) return;
    ok &= (d_field_min(xm(a)) - k >= 1) | d_is0(a.re) | d_is0(a.im);
    ok &= k > -1023;                                    // not 0 (nor subnormal)
    a.re = d_shift(a.re, -k);
    a.im = d_shift(a.im, -k);
    a.e += k;
}

// xr_mul by the integer products
FSG_DEV xc xs_mul(xc a, xc b) {
    double2 m = cmul_soft(xm(a), xm(b));
    int e = (int)((unsigned)a.e + (unsigned)b.e);
    if (xr_need_renorm_c(m)) return xr_normalize_c(m, e);
    return xc_make(m.x, m.y, e);
}

// ---------------------------------------------------------------------------
// |z| < r as hypot(z) < r decides it, from upper words: |z|^2 = q 2^2e with q in
// [1, 8) known to a part in 2^18 (mag_of: the words as floats, cut to 20 bits, on
// the larger part's exponent), against r^2 on the same exponent.  -1: too close,
// or out of the normal range (abs_cmp and hypot decide, fsg_num.cuh).
// ---------------------------------------------------------------------------
struct MagF { float q; int e; bool ok; };
FSG_DEV MagF mag_of(double2 z, int ze) {
    const unsigned hx = d_hi(z.x) & 0x7fffffffu, hy = d_hi(z.y) & 0x7fffffffu, m = max(hx, hy);
    const unsigned base = (m & 0x7ff00000u) - (127u << 20);
    const float x = __int_as_float(max((int)(hx - base), 0) << 3);
    const float y = __int_as_float(max((int)(hy - base), 0) << 3);
    MagF a;
    a.q = x * x + y * y;
    a.e = (int)(m >> 20) - 1023 + ze;
    a.ok = m >= 0x00100000u && m < 0x7ff00000u;
    return a;
}
FSG_DEV int mag_lt(const MagF &a, double r) {
    const unsigned h = d_hi(r);
    if (d_is0(r)) return 0;                               // never below 0
    if (!a.ok || h < 0x00100000u || h >= 0x7ff00000u) return -1;
    const int d = (int)(h >> 20) - 1023 - a.e;
    if (d >= 3) return 1;                                 // |z| < 2^(e + 1.5)
    // (near the end of the doubles' range the loops compare the rounded value)
    if (a.e < -1000) return -1;
    if (d <= -2) return 0;                                // r < 2^(e - 1)
    const float f = __int_as_float((int)((h & 0x000fffffu) << 3 | (unsigned)(d + 127) << 23));
    const float f2 = f * f;
    if (a.q * (1.f + 0x1p-17f) < f2) return 1;
    if (a.q > f2 * (1.f + 0x1p-17f)) return 0;
    return -1;
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
