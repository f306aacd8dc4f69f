// Host check of fractalshades_gb300/csrc/fsg_soft.cuh: a product that keeps
// `ok` has the bits of the double product, and the exponent thresholds decide
// only what the double comparison decides.  Operands: random, with few
// mantissa bits (exact products, ties), next to powers of two, at and beyond
// the ends of the accepted exponents, zeros, subnormals, infinities and NaNs.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
static inline long long __double_as_longlong(double d) { long long x; memcpy(&x, &d, 8); return x; }
static inline double __longlong_as_double(long long x) { double d; memcpy(&d, &x, 8); return d; }
static inline double __hiloint2double(int hi, int lo) {
    return __longlong_as_double((long long)((unsigned long long)(unsigned)hi << 32 | (unsigned)lo));
}
static inline int __float_as_int(float f) { int x; memcpy(&x, &f, 4); return x; }
static inline float __int_as_float(int x) { float f; memcpy(&f, &x, 4); return f; }
static inline unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s) {
    return (unsigned)(((((unsigned long long)hi << 32) | lo) << (s & 31)) >> 32);
}
static inline unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned s) {
    return (unsigned)((((unsigned long long)hi << 32) | lo) >> (s & 31));
}
using std::max;
using std::min;
#ifndef __noinline__
#define __noinline__ __attribute__((noinline))
#endif
#include "../../fractalshades_gb300/csrc/fsg_soft.cuh"

static bool same(double a, double b) { return (std::isnan(a) && std::isnan(b)) || dbits(a) == dbits(b); }

int main(int argc, char **argv) {
    const long cases = argc > 1 ? atol(argv[1]) : 2000000;
    std::mt19937_64 g(11);
    const double special[] = {0., -0., 1., -1., INFINITY, -INFINITY, NAN, 4.9e-324, 1e-310,
                              0x1p-480, 0x1p-481, 0x1.fffffffffffffp479, 0x1p480, 0x1p-1022, 1.7e308};
    auto draw = [&]() {
        const int kind = (int)(g() % 10);
        if (kind == 0) return special[g() % 15];
        unsigned long long m = g() >> 12;                            // 52 bits
        if (kind < 4) m &= ~0ULL << (g() % 52);                      // few low bits
        if (kind == 4) m = (g() % 16);                               // next above a power of two
        if (kind == 5) m = 0xfffffffffffffULL - (g() % 16);          // next below
        const int e = kind < 8 ? (int)(g() % 200) - 100 : (int)(g() % 1100) - 550;
        double d = __longlong_as_double((long long)((unsigned long long)(e + 1023) << 52 | m));
        return (g() & 1) ? -d : d;
    };
    long bad = 0, kept = 0, open = 0;
    auto miss = [&](const char *what, double x, double y) {
        if (bad++ < 5) printf("%s(%a, %a)\n", what, x, y);
    };
    for (long i = 0; i < cases; i++) {
        const double x = draw(), y = draw(), u = draw(), v = draw();
        volatile double xy = x * y, xx = x * x, x2y = 2. * x * y;
        if (dfac_ok(x) && dfac_ok(y)) {
            bool ok = true;
            const double p = dfac_mul(dfac_of(x), dfac_of(y), ok);
            if (ok && !same(p, xy)) miss("dfac_mul", x, y);
            ok ? kept++ : open++;
            ok = true;
            const double s = dfac_mul(dfac_of(x), dfac_of(x), ok);
            if (ok && !same(s, xx)) miss("square", x, x);
            ok = true;
            const double t = dfac_mul(dfac_of(x, 1), dfac_of(y), ok);
            if (ok && !same(t, x2y)) miss("twice", x, y);
        }
        if (dfac_ok(x) && dfac_ok(y)) {
            const double k = (double)(1 + g() % 40);
            volatile double kx = k * x;
            if (!same(dfac_mul_ties(dfac_of(x), dfac_of(y)), xy)) miss("dfac_mul_ties", x, y);
            if (!same(dfac_mul_ties(dfac_of(k), dfac_of(x)), kx)) miss("dfac_mul_ties", k, x);
        }
        if (dfac_ok0(x) && dfac_ok0(y)) {
            bool ok = true;
            const double p = dfac_mul0(dfac_of0(x), dfac_of0(y), ok);
            if (ok && !same(p, xy)) miss("dfac_mul0", x, y);
        }
        if (dfac_ok(cx(x, y)) && dfac_ok(cx(u, v))) {
            bool ok = true;
            const double2 p = cfac_mul(cfac_of(cx(x, y)), cfac_of(cx(u, v)), ok);
            const double2 q = cmul(cx(x, y), cx(u, v));
            if (ok && (!same(p.x, q.x) || !same(p.y, q.y))) miss("cfac_mul", x, u);
            ok = true;
            const double2 r = cfac_sq(cfac_of(cx(x, y)), ok), w = csq(cx(x, y));
            if (ok && (!same(r.x, w.x) || !same(r.y, w.y))) miss("cfac_sq", x, y);
        }
        // products of parts of any size, and with zero parts
        if (cfac_ok<false>(cx(x, y), cx(u, v))) {
            bool ok = true;
            const double2 p = cfac_mul(cfac_of(cx(x, y)), cfac_of(cx(u, v)), ok);
            const double2 q = cmul(cx(x, y), cx(u, v));
            if (ok && (!same(p.x, q.x) || !same(p.y, q.y))) miss("cfac_ok", x, u);
        }
        if (cfac_ok<true>(cx(x, 0.), cx(u, v))) {
            bool ok = true;
            const double2 p = cfac_mul0(cfac_of0(cx(x, 0.)), cfac_of(cx(u, v)), ok);
            const double2 q = cmul(cx(x, 0.), cx(u, v));
            if (ok && (!same(p.x, q.x) || !same(p.y, q.y))) miss("cfac_ok0", x, u);
        }
        // p 2^ep + q 2^eq on one frame: the rounded sums on p's frame, for q that
        // stays normal there
        {
            const int ep = (int)(g() % 4000) - 2000, d = (int)(g() % 300) - 150;
            const double2 p = cx(std::ldexp(x, -(int)(g() % 40)), y), q = cx(u, v);
            if (dfac_ok0(p.x) & dfac_ok0(p.y) & dfac_ok0(u) & dfac_ok0(v)) {
                bool ok = true;
                xc r = frame_add(p, ep, q, ep + d, ok);
                volatile double sx = p.x + std::ldexp(u, d), sy = p.y + std::ldexp(v, d);
                if (!ok) miss("frame_add range", p.x, u);
                if (std::ldexp(r.re, r.e - ep) != sx || std::ldexp(r.im, r.e - ep) != sy) miss("frame_add", p.x, u);
                const xc before = r;
                ok = true;
                frame_renorm(r, ok);
                if (ok && (std::ldexp(r.re, r.e - before.e) != before.re || std::ldexp(r.im, r.e - before.e) != before.im))
                    miss("frame_renorm", before.re, before.im);
            }
        }
        // |z| < r from upper words
        {
            const double h = std::hypot(x, y);
            const MagF m = mag_of(cx(x, y), 0);
            if (std::isnan(h)) continue;
            for (double r : {std::fabs(u), h, std::nextafter(h, INFINITY), h * 1.00001, h * 0.99999, h * 3., h * 0.3, 0.}) {
                const int lt = mag_lt(m, r);
                if (lt >= 0 && lt != (h < r ? 1 : 0)) miss("mag_lt", h, r);
            }
        }
        // thresholds: t itself a square, and |z| drawn near its root too
        const double t = u * u, near = std::sqrt(t) * (1. + ((int)(g() % 5) - 2) * 0x1p-52);
        const SqBound b = fsg_sq_bound(t);
        for (double a : {x, near, near * 0.70710678118654752, near * 0.9, near * 0.5, 0.})
            for (double c : {y, a, near * 0.43588989435406736, 0.}) {
                volatile double s = a * a + c * c;
                if (d_abs2_gt(cx(a, c), t, b) != (s > t)) miss("d_abs2_gt", a, t);
                if (d_abs2_lt(cx(a, c), t, b) != (s < t)) miss("d_abs2_lt", a, t);
            }
    }
    printf("%ld cases, %ld products kept, %ld open, %ld mismatches\n", cases, kept, open, bad);
    return bad != 0 || kept < cases / 10;
}
