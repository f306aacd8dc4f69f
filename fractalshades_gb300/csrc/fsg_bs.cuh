// fsg_bs.cuh -- the Burning Ship family perturbation loop, templated on the
// real type of the deltas:
//   * double -- the reference's standard branch (instantiated in
//     fsg_perturb_bs64.cu, compiled without FMA contraction: one rounding per
//     operation in the order of the reference source);
//   * fr -- FP32 mantissa + int32 exponent (instantiated in fsg_perturb_bs32.cu):
//     no underflow at any depth and FP32-pipe arithmetic instead of GB300's
//     slow FP64 pipe; results within FP32 rounding of the double form.
// perturbation.py:1406-1811 (numba_cycles_perturb_BS, numba_iterate_BS,
// apply_BLA_BS, apply_BLA_deriv_BS) with the closures of
// models/burning_ship.py:19-60 (diffabs and its derivatives), 535-619
// (_p_iter_zn) and 622-859 (_p_iter_hessian).
#pragma once
#include "fsg_internal.cuh"

// Whether ref_BLA_get can admit any dz at start index w >> 3: radii never
// grow with the stage (combine_BLA, combine_BLA_BS: r <= r of the first child,
// perturbation.py:2023-2024, 2104-2105) and 0 < r is strict, so a stage-3
// radius of 0 -- at the orbit's critical point, where A = 2 Z = 0 -- rules
// every stage out, and |dz| need not be computed for the search.
__device__ __forceinline__ bool bla_possible(const RefDev &R, int w) {
    const int i3 = 2 * (w >> FSG_STG_COMPRESSED);
    return i3 < R.bla_len && d_sq_gt(__ldg(&R.rbla[i3]), 0.);
}

// perturbation.py:2116-2170 ref_BLA_get on dz itself: returns the step (0 if
// none) and the table index of the accepted entry.  The reference tests
// abs(dz) < r, a hypot, against each candidate radius; mag_lt (fsg_soft.cuh)
// decides all but about one in 10^5 from upper words, without FP64.
// The search of ref_BLA_get with `lt(r)` for abs(dz) < r: the step and its index
template <class LT>
__device__ __forceinline__ int bla_search(const RefDev &R, int w, int &ib, LT lt) {
    int it = w >> FSG_STG_COMPRESSED;
    int stages = FSG_STG_COMPRESSED;
    for (int st = FSG_STG_COMPRESSED; st < R.stages; st++) {
        stages = st;
        if (it & 1) break;
        it >>= 1;
    }
    const int invalid_step = R.first_invalid - w;
    for (int stg = stages; stg >= FSG_STG_COMPRESSED; stg--) {
        const int step = 1 << stg;
        if (step >= invalid_step) continue;
        const int idx = 2 * (w >> FSG_STG_COMPRESSED) + ((1 << (stg - FSG_STG_COMPRESSED)) - 1);
        if (lt(__ldg(&R.rbla[idx]))) { ib = idx; return step; }
    }
    return 0;
}
// |z| < r where upper words leave it open: abs_cmp, then hypot (a: |z|^2 on z's own
// scale, h: hypot(z), each once per lookup)
struct BLAExact { AbsScaled a; double h; bool has; };
static __device__ __noinline__ int bla_exact_lt(double2 z, double r, BLAExact &x) {
    if (!x.has) { x.a = abs_scaled(z); x.h = -1.; x.has = true; }
    const int lt = abs_cmp(x.a, r);
    if (lt >= 0) return lt;
    if (x.h < 0.) x.h = hypot(z.x, z.y);
    return x.h < r;
}
__device__ __forceinline__ int bla_lookup_z(const RefDev &R, double2 z, int w, int &ib) {
    const MagF a = mag_of(z, 0);
    BLAExact x;
    x.has = false;
    return bla_search(R, w, ib, [&](double r) {
        const int lt = mag_lt(a, r);
        return lt >= 0 ? lt : bla_exact_lt(z, r, x);
    });
}
// the same for dz = z, an Xrange value whose standard value is compared
__device__ __forceinline__ int bla_lookup_x(const RefDev &R, xc z, int w, int &ib) {
    const MagF a = mag_of(xm(z), z.e);
    BLAExact x;
    x.has = false;
    return bla_search(R, w, ib, [&](double r) {
        const int lt = mag_lt(a, r);
        return lt >= 0 ? lt : bla_exact_lt(xr_to_std(z), r, x);
    });
}

// ---------------------------------------------------------------------------
// fr: a real m * 2^e with an FP32 mantissa, |m| in [1, 2), or m = 0 (e =
// FR_ZERO_E).  Every operation rounds the mantissa once (FP32) and keeps the
// exponent exact.
// ---------------------------------------------------------------------------
struct fr { float m; int e; };
#define FR_ZERO_E (-(1 << 29))

FSG_DEV fr fr_zero() { fr r; r.m = 0.f; r.e = FR_ZERO_E; return r; }
// normalise m * 2^e for finite m (0 and subnormal mantissas give 0): the
// biased exponent of m moves to e and m's own is set to 0 (bit operations)
FSG_DEV fr fr_norm(float m, int e) {
    const int bits = __float_as_int(m);
    const int b = (bits >> 23) & 0xff;
    fr r;
    r.m = __int_as_float((bits & 0x807fffff) | 0x3f800000);
    r.e = e + (b - 127);
    if (b == 0) r = fr_zero();
    return r;
}
FSG_DEV fr fr_from_d(double x) {
    const long long bits = __double_as_longlong(x);
    const int be = (int)((bits >> 52) & 0x7ff);
    if (be == 0) {
        if (x == 0.) return fr_zero();
        int e; double f = frexp(x, &e);            // subnormal double
        return fr_norm((float)(2. * f), e - 1);
    }
    // the mantissa in [1, 2) with the sign of x; its FP32 rounding may give 2
    const double m = __longlong_as_double((bits & 0x800fffffffffffffLL) | 0x3ff0000000000000LL);
    return fr_norm((float)m, be - 1023);
}
FSG_DEV double fr_to_d(fr a) { return a.m == 0.f ? 0. : ldexp_d((double)a.m, a.e); }
// 2^-d for d >= 0 (0 from d = 127 on)
FSG_DEV float fr_p2n(int d) { return __int_as_float((127 - min(d, 127)) << 23); }

// Branch-free: the operand of larger exponent (a zero has the smallest) takes
// the other scaled by 2^-d in one FMA.  From d = 61 on the scaled term is
// below half an ulp and the sum is the larger operand itself.
FSG_DEV fr operator+(fr a, fr b) {
    const bool ge = a.e >= b.e;
    const float mb = ge ? a.m : b.m, ms = ge ? b.m : a.m;
    const int eb = ge ? a.e : b.e, d = ge ? a.e - b.e : b.e - a.e;
    return fr_norm(fmaf(ms, fr_p2n(d), mb), eb);
}
FSG_DEV fr operator-(fr a) { a.m = -a.m; return a; }
FSG_DEV fr operator-(fr a, fr b) { return a + (-b); }
FSG_DEV fr operator*(fr a, fr b) {
    fr r; r.m = a.m * b.m; r.e = a.e + b.e;              // |m| in [1, 4) or 0
    if (fabsf(r.m) >= 2.f) { r.m *= 0.5f; r.e += 1; }
    if (r.m == 0.f) r = fr_zero();
    return r;
}
// product by a literal constant (the closures' 2. * x): FP32 only, exact for
// the powers of two the loop uses
FSG_DEV fr operator*(double s, fr b) {
    if (s == 2. || s == -2.) {
        if (b.m != 0.f) b.e += 1;
        if (s < 0.) b.m = -b.m;
        return b;
    }
    return fr_norm((float)s * b.m, b.e);
}
FSG_DEV fr &operator+=(fr &a, fr b) { a = a + b; return a; }

// xf: the reference's float64 Xrange record (numba_xr.py), the real type of
// the Xrange branch.  Constants are the unnormalised records {x, 0}, so that a
// constant times a record rounds as the reference's float * Xrange.
FSG_DEV xf operator+(xf a, xf b) { return xf_add(a, b); }
FSG_DEV xf operator-(xf a) { a.m = -a.m; return a; }
FSG_DEV xf operator-(xf a, xf b) { return xf_sub(a, b); }
FSG_DEV xf operator*(xf a, xf b) { return xf_mul(a, b); }
FSG_DEV xf operator*(double s, xf b) { return xf_mul_s(s, b); }
FSG_DEV xf &operator+=(xf &a, xf b) { a = a + b; return a; }

// the operations the loop needs, for every real type
FSG_DEV double to_d(double x) { return x; }
FSG_DEV double to_d(fr x) { return fr_to_d(x); }
FSG_DEV double to_d(xf x) { return xf_to_std(x); }
template <class T> FSG_DEV T from_d(double x);
template <> FSG_DEV double from_d<double>(double x) { return x; }
template <> FSG_DEV fr from_d<fr>(double x) { return fr_from_d(x); }
template <> FSG_DEV xf from_d<xf>(double x) { return xr_from_r(x); }      // to_Xrange_scalar
// a literal constant (0, +-1, +-2) of the loop's real type, without FP64
template <class T> FSG_DEV T cst(float x);
template <> FSG_DEV double cst<double>(float x) { return (double)x; }
template <> FSG_DEV fr cst<fr>(float x) { return fr_norm(x, 0); }
template <> FSG_DEV xf cst<xf>(float x) { return xf_make((double)x, 0); }
// m * 2^e from a mantissa and an exponent (the Xrange form of c)
template <class T> FSG_DEV T from_me(double m, int e);
template <> FSG_DEV double from_me<double>(double m, int e) { return ldexp_d(m, e); }
template <> FSG_DEV fr from_me<fr>(double m, int e) {
    fr r = fr_from_d(m);
    if (r.m != 0.f) r.e += e;
    return r;
}
template <> FSG_DEV xf from_me<xf>(double m, int e) { return xf_make(m, e); }
FSG_DEV bool ge0(double x) { return d_ge0(x); }
FSG_DEV bool ge0(fr x) { return x.m >= 0.f; }
FSG_DEV bool ge0(xf x) { return xf_ge_s(x, 0.); }
FSG_DEV bool le0(double x) { return d_le0(x); }
FSG_DEV bool le0(fr x) { return x.m <= 0.f; }
FSG_DEV bool le0(xf x) { return xf_le_s(x, 0.); }
FSG_DEV double absT(double x) { return d_abs(x); }
FSG_DEV fr absT(fr x) { x.m = fabsf(x.m); return x; }
FSG_DEV xf absT(xf x) { x.m = fabs(x.m); return x; }
// sgn with 0 mapped to +1 (burning_ship.py:12-17)
FSG_DEV double sgnT(double x) { return d_lt0(x) ? -1. : 1.; }
FSG_DEV fr sgnT(fr x) { fr r; r.m = x.m < 0.f ? -1.f : 1.f; r.e = 0; return r; }
FSG_DEV xf sgnT(xf x) { return xf_make(xf_lt_s(x, 0.) ? -1. : 1., 0); }
// |a| <= |b|
FSG_DEV bool abs_le(double a, double b) { return d_abs_le(a, b); }
FSG_DEV bool abs_le(xf a, xf b) { a.m = fabs(a.m); b.m = fabs(b.m); return xf_le(a, b); }
FSG_DEV bool abs_le(fr a, fr b) {
    if (a.m == 0.f) return true;
    if (b.m == 0.f) return false;
    return a.e != b.e ? a.e < b.e : fabsf(a.m) <= fabsf(b.m);
}

// |(x, y)| as s * 2^e, s in [1, 2 sqrt 2], in FP32 (z = false: (0, 0))
struct fr_mod { float s; int e; bool z; };
FSG_DEV fr_mod fr_modulus2(fr x, fr y, bool squared) {
    const int e = max(x.e, y.e);
    const float mx = x.m * fr_p2n(e - x.e), my = y.m * fr_p2n(e - y.e);
    const float q = fmaf(mx, mx, my * my);
    fr_mod r; r.s = squared ? q : sqrtf(q); r.e = squared ? 2 * e : e;
    r.z = x.m == 0.f && y.m == 0.f;
    return r;
}
// v * 2^d as a float, d in [-3, 0]
FSG_DEV float fr_scale_small(float v, int d) { return v * __int_as_float((127 + d) << 23); }

// The double-precision forms of the two comparisons below, for the rare
// near-ties: out of line so that the compiler does not evaluate them ahead
// of the branch on every call.
static __device__ __noinline__ bool fr_escaped_exact(fr X, fr Y, double M2) {
    const double Xd = fr_to_d(X), Yd = fr_to_d(Y);
    return Xd * Xd + Yd * Yd > M2;
}
static __device__ __noinline__ bool fr_below_exact(fr xn, fr yn, double r) {
    return hypot(fr_to_d(xn), fr_to_d(yn)) < r;
}

// The escape test |z|^2 > M2 of the loop (perturbation.py:1636-1639) with z in
// fr: decided in FP32 unless within 2^-18 of the bound, where the double form
// of the reference decides (so that the outcome is the FP64 one of the same
// fr values).
FSG_DEV bool fr_escaped(fr X, fr Y, fr M2f, double M2) {
    const fr_mod q = fr_modulus2(X, Y, true);           // s in [1, 8)
    if (q.z) return false;                              // M2 > 0
    const int d = q.e - M2f.e;
    if (d >= 1) return true;                            // >= 2 > M2 mantissa
    if (d <= -4) return false;                          // < 0.5
    const float t = fr_scale_small(q.s, d);
    if (fabsf(t - M2f.m) > M2f.m * 0x1p-18f) return t > M2f.m;
    return fr_escaped_exact(X, Y, M2);
}

// |dz| < r for a BLA radius r (double r, its fr copy rm * 2^re), the
// comparison of ref_BLA_get (perturbation.py:2116-2170) in FP32 unless within
// 2^-18 of r, where the double form decides.
FSG_DEV bool fr_below(const fr_mod &a, fr xn, fr yn, float rm, int re, double r) {
    if (rm == 0.f) return false;                        // r = 0
    if (a.z) return true;                               // 0 < r
    const int d = a.e - re;
    if (d >= 1) return false;                           // >= 2 > rm
    if (d <= -2) return true;                           // < 0.71 < rm
    const float t = fr_scale_small(a.s, d);
    if (fabsf(t - rm) > rm * 0x1p-18f) return t < rm;
    return fr_below_exact(xn, yn, r);
}

// ref_BLA_get in the loop's real type: double |dz| against the double radii,
// or the FP32 modulus against their fr copies
template <class T> struct BLAGet;
template <> struct BLAGet<double> {
    static FSG_DEV int get(const RefDev &R, double xn, double yn, int w, int &ib) {
        return bla_possible(R, w) ? bla_lookup_z(R, cx(xn, yn), w, ib) : 0;
    }
};
template <> struct BLAGet<fr> {
    static FSG_DEV int get(const RefDev &R, fr xn, fr yn, int w, int &ib) {
        if (!bla_possible(R, w)) return 0;
        int it = w >> FSG_STG_COMPRESSED;
        int stages = FSG_STG_COMPRESSED;
        for (int s = FSG_STG_COMPRESSED; s < R.stages; s++) {
            stages = s;
            if (it & 1) break;
            it >>= 1;
        }
        const fr_mod a = fr_modulus2(xn, yn, false);
        const int invalid_step = R.first_invalid - w;
        for (int stg = stages; stg >= FSG_STG_COMPRESSED; stg--) {
            const int step = 1 << stg;
            if (step >= invalid_step) continue;
            const int idx = 2 * (w >> FSG_STG_COMPRESSED) + ((1 << (stg - FSG_STG_COMPRESSED)) - 1);
            const int2 rf = __ldg(&R.bs_rf[idx]);
            if (fr_below(a, xn, yn, __int_as_float(rf.x), rf.y, __ldg(&R.rbla[idx]))) {
                ib = idx;
                return step;
            }
        }
        return 0;
    }
};

// v * 2^k (k = 0: v)
FSG_DEV double scale2(double v, int k) { return k == 0 ? v : ldexp_d(v, k); }
FSG_DEV fr scale2(fr v, int k) { if (v.m != 0.f) v.e += k; return v; }
FSG_DEV xf scale2(xf v, int k) { v.e += k; return v; }

// ref_BLA_get on the Xrange branch: the standard values of the deltas (0
// below the double range, perturbation.py:1520-1527)
template <> struct BLAGet<xf> {
    static FSG_DEV int get(const RefDev &R, xf xn, xf yn, int w, int &ib) {
        return bla_possible(R, w) ? bla_lookup_z(R, cx(xf_to_std(xn), xf_to_std(yn)), w, ib)
                                  : 0;
    }
};

// Reads of the reference's tables in the loop's real type: the double
// tables themselves, or their fr copies (orbit values from the Xrange side
// table where the orbit holds one)
template <class T> struct BSRef;
template <> struct BSRef<double> {
    static FSG_DEV void orbit(const RefDev &R, int w, double &X, double &Y) {
        double2 z = __ldg(&R.Zn[w]); X = z.x; Y = z.y;
    }
    static FSG_DEV void hess(const RefDev &R, int w, double &a, double &b, double &c, double &d) {
        a = __ldg(&R.dXa[w]); b = __ldg(&R.dXb[w]); c = __ldg(&R.dYa[w]); d = __ldg(&R.dYb[w]);
    }
    static FSG_DEV void bla(const RefDev &R, int ib, double M[8]) {
        const double *p = R.Mbla_bs + 8 * ib;
        for (int k = 0; k < 8; k++) M[k] = __ldg(p + k);
    }
};
template <> struct BSRef<fr> {
    static FSG_DEV fr lo(int4 v) { fr r; r.m = __int_as_float(v.x); r.e = v.y; return r; }
    static FSG_DEV fr hi(int4 v) { fr r; r.m = __int_as_float(v.z); r.e = v.w; return r; }
    static FSG_DEV void orbit(const RefDev &R, int w, fr &X, fr &Y) {
        int4 v = __ldg(&R.bs_Zf[w]); X = lo(v); Y = hi(v);
    }
    static FSG_DEV void hess(const RefDev &R, int w, fr &a, fr &b, fr &c, fr &d) {
        int4 p = __ldg(&R.bs_hf[2 * w]), q = __ldg(&R.bs_hf[2 * w + 1]);
        a = lo(p); b = hi(p); c = lo(q); d = hi(q);
    }
    static FSG_DEV void bla(const RefDev &R, int ib, fr M[8]) {
        for (int k = 0; k < 4; k++) {
            int4 v = __ldg(&R.bs_blaf[4 * ib + k]);
            M[2 * k] = lo(v); M[2 * k + 1] = hi(v);
        }
    }
};

// The Xrange branch: ensure_xr_BS (perturbation.py:2182-2193) -- the side
// table's value where the orbit holds one, else the standard value as a
// record; the Xrange Jacobian paths; the BLA coefficients as float64 (the
// reference multiplies them float * Xrange: unnormalised records {M, 0})
template <> struct BSRef<xf> {
    static FSG_DEV bool table(const RefDev &R, int w, xf &X, xf &Y) {
        const int s = (R.n_xr > 0 && w < R.len) ? __ldg(&R.xr_slot[w]) : -1;
        if (s < 0) return false;
        const double *m = (const double *)R.xr_m;
        X = xf_make(__ldg(&m[s]), __ldg(&R.xr_e[s]));
        Y = xf_make(__ldg(&m[R.n_xr + s]), __ldg(&R.xr_e[R.n_xr + s]));
        return true;
    }
    static FSG_DEV void orbit(const RefDev &R, int w, xf &X, xf &Y) {
        if (!table(R, w, X, Y)) {
            const double2 z = __ldg(&R.Zn[w]);
            X = xr_from_r(z.x); Y = xr_from_r(z.y);
        }
    }
    static FSG_DEV void hess(const RefDev &R, int w, xf &a, xf &b, xf &c, xf &d) {
        const int L = R.len + 1;
        a = xf_make(__ldg(&R.bs_xpm[w]), __ldg(&R.bs_xpe[w]));
        b = xf_make(__ldg(&R.bs_xpm[L + w]), __ldg(&R.bs_xpe[L + w]));
        c = xf_make(__ldg(&R.bs_xpm[2 * L + w]), __ldg(&R.bs_xpe[2 * L + w]));
        d = xf_make(__ldg(&R.bs_xpm[3 * L + w]), __ldg(&R.bs_xpe[3 * L + w]));
    }
    static FSG_DEV void bla(const RefDev &R, int ib, xf M[8]) {
        const double *p = R.Mbla_bs + 8 * ib;
        for (int k = 0; k < 8; k++) M[k] = xf_make(__ldg(p + k), 0);
    }
};

// burning_ship.py:19-60 diffabs(X, x) = |X + x| - |X| and its derivatives
// 2. * x and 1. * x of the closures in their real type: for a double, the
// doubling on the exponent bits and x itself (a NaN or inf takes the
// product, out of line) -- the same bits with no FP64 instruction
FSG_DEV double twice_t(double x) { return d_twice(x); }
FSG_DEV fr twice_t(fr x) { return 2. * x; }
FSG_DEV xf twice_t(xf x) { return 2. * x; }
static __device__ __noinline__ double d_one_full(double x) { return 1. * x; }
FSG_DEV double one_t(double x) { return d_nonfinite(x) ? d_one_full(x) : x; }
FSG_DEV fr one_t(fr x) { return 1. * x; }
FSG_DEV xf one_t(xf x) { return 1. * x; }
template <class T> FSG_DEV T diffabs(T X, T x) {
    if (ge0(X)) { if (ge0(X + x)) return one_t(x); else return -(twice_t(X) + x); }
    else { if (le0(X + x)) return -x; else return (twice_t(X) + x); }
}
template <class T> FSG_DEV T ddiffabsdX(T X, T x) {
    if (ge0(X)) { if (ge0(X + x)) return cst<T>(0.f); else return cst<T>(-2.f); }
    else { if (le0(X + x)) return cst<T>(0.f); else return cst<T>(2.f); }
}
template <class T> FSG_DEV T ddiffabsdx(T X, T x) {
    if (ge0(X)) { if (ge0(X + x)) return cst<T>(1.f); else return cst<T>(-1.f); }
    else { if (le0(X + x)) return cst<T>(-1.f); else return cst<T>(1.f); }
}

// burning_ship.py:535-619 _p_iter_zn
template <class T>
FSG_DEV void bs_zn(int flavor, T &xn, T &yn, T X, T Y, T a, T b) {
    T nx, ny;
    if (flavor == 1) {
        T ref_xyn = X * Y;
        nx = xn * (xn + twice_t(X)) - yn * (yn + twice_t(Y)) + a;
        ny = twice_t(diffabs(ref_xyn, xn * yn + xn * Y + yn * X)) - b;
    } else if (flavor == 2) {
        nx = xn * (xn + twice_t(X)) - yn * (yn + twice_t(Y)) + a;
        ny = twice_t(X * diffabs(Y, yn) + xn * absT(Y + yn)) - b;
    } else if (flavor == 3) {
        nx = xn * (xn + twice_t(X)) - Y * diffabs(Y, yn) - yn * absT(Y + yn) + a;
        ny = twice_t(X * yn + Y * xn + xn * yn) - b;
    } else if (flavor == 4) {
        T q = X * X - Y * Y;
        nx = diffabs(q, xn * (xn + twice_t(X)) - yn * (yn + twice_t(Y))) + a;
        ny = twice_t(X * yn + Y * xn + xn * yn) - b;
    } else {
        T ref_xyn = X * Y, q = X * X - Y * Y;
        nx = diffabs(q, xn * (xn + twice_t(X)) - yn * (yn + twice_t(Y))) + a;
        ny = twice_t(diffabs(ref_xyn, xn * yn + xn * Y + yn * X)) - b;
    }
    xn = nx; yn = ny;
}

// burning_ship.py:622-859 _p_iter_hessian, h = (dxnda, dxndb, dynda, dyndb)
template <class T>
FSG_DEV void bs_hess(int flavor, T h[4], T xn, T yn, T X, T Y, T Xa, T Xb, T Ya, T Yb) {
    T xa = h[0], xb = h[1], ya = h[2], yb = h[3];
    T nxa, nxb, nya, nyb;
    if (flavor == 1 || flavor == 5) {
        T opX = X * Y;
        T dXa = Xa * Y + X * Ya, dXb = Xb * Y + X * Yb;
        T opx = xn * yn + xn * Y + yn * X;
        T dxa = xa * yn + xn * ya + xa * Y + xn * Ya + ya * X + yn * Xa;
        T dxb = xb * yn + xn * yb + xb * Y + xn * Yb + yb * X + yn * Xb;
        T dX = ddiffabsdX(opX, opx), dx = ddiffabsdx(opX, opx);
        nya = twice_t(dX * dXa + dx * dxa);
        nyb = twice_t(dX * dXb + dx * dxb);
        if (flavor == 1) {
            nxa = twice_t((X + xn) * xa + Xa * xn) - twice_t((Y + yn) * ya + Ya * yn);
            nxb = twice_t((X + xn) * xb + Xb * xn) - twice_t((Y + yn) * yb + Yb * yn);
        } else {
            T opX2 = X * X - Y * Y;
            T dXa2 = twice_t(X * Xa - Y * Ya), dXb2 = twice_t(X * Xb - Y * Yb);
            T opx2 = xn * (xn + twice_t(X)) - yn * (yn + twice_t(Y));
            T dxa2 = xa * (xn + twice_t(X)) + xn * (xa + twice_t(Xa)) - ya * (yn + twice_t(Y)) - yn * (ya + twice_t(Ya));
            T dxb2 = xb * (xn + twice_t(X)) + xn * (xb + twice_t(Xb)) - yb * (yn + twice_t(Y)) - yn * (yb + twice_t(Yb));
            T dX2 = ddiffabsdX(opX2, opx2), dx2 = ddiffabsdx(opX2, opx2);
            nxa = dX2 * dXa2 + dx2 * dxa2;
            nxb = dX2 * dXb2 + dx2 * dxb2;
        }
    } else if (flavor == 2) {
        T da = diffabs(Y, yn), dX = ddiffabsdX(Y, yn), dx = ddiffabsdx(Y, yn);
        T Yy = Y + yn, ab = absT(Yy), sg = sgnT(Yy);
        nxa = twice_t(((X + xn) * xa + Xa * xn) - ((Y + yn) * ya + Ya * yn));
        nxb = twice_t(((X + xn) * xb + Xb * xn) - ((Y + yn) * yb + Yb * yn));
        nya = twice_t(Xa * da + X * (dX * Ya + dx * ya) + xa * ab + xn * sg * (Ya + ya));
        nyb = twice_t(Xb * da + X * (dX * Yb + dx * yb) + xb * ab + xn * sg * (Yb + yb));
    } else if (flavor == 3) {
        T da = diffabs(Y, yn), dX = ddiffabsdX(Y, yn), dx = ddiffabsdx(Y, yn);
        T Yy = Y + yn, ab = absT(Yy), sg = sgnT(Yy);
        nxa = xa * (xn + twice_t(X)) + xn * (xa + twice_t(Xa)) - Ya * da - Y * (Ya * dX + ya * dx)
              - ya * ab - yn * sg * (Ya + ya);
        nxb = xb * (xn + twice_t(X)) + xn * (xb + twice_t(Xb)) - Yb * da - Y * (Yb * dX + yb * dx)
              - yb * ab - yn * sg * (Yb + yb);
        nya = twice_t(Xa * yn + X * ya + Ya * xn + Y * xa + xa * yn + xn * ya);
        nyb = twice_t(Xb * yn + X * yb + Yb * xn + Y * xb + xb * yn + xn * yb);
    } else {
        T opX = X * X - Y * Y;
        T dXa = twice_t(X * Xa - Y * Ya), dXb = twice_t(X * Xb - Y * Yb);
        T opx = xn * (xn + twice_t(X)) - yn * (yn + twice_t(Y));
        T dxa = xa * (xn + twice_t(X)) + xn * (xa + twice_t(Xa)) - ya * (yn + twice_t(Y)) - yn * (ya + twice_t(Ya));
        T dxb = xb * (xn + twice_t(X)) + xn * (xb + twice_t(Xb)) - yb * (yn + twice_t(Y)) - yn * (yb + twice_t(Yb));
        T dX = ddiffabsdX(opX, opx), dx = ddiffabsdx(opX, opx);
        nxa = dX * dXa + dx * dxa;
        nxb = dX * dXb + dx * dxb;
        nya = twice_t(Xa * yn + X * ya + Ya * xn + Y * xa + xa * yn + xn * ya);
        nyb = twice_t(Xb * yn + X * yb + Yb * xn + Y * xb + xb * yn + xn * yb);
    }
    h[0] = nxa; h[1] = nxb; h[2] = nya; h[3] = nyb;
}

// ---------------------------------------------------------------------------
// Frame form of the fr loop.  The delta pair shares one exponent and the
// Hessian another:  (xn, yn) = (ux, uy) 2^E,  (dxnda, dxndb, dynda, dyndb) =
// h 2^F,  with (a, b) 2^-E kept as (cux, cuy).  A step then runs the closures'
// formulas (burning_ship.py:535-859) in plain FP32: the orbit values X, Y are
// floats (the fa table), products of two deltas carry the factor s = 2^E (0
// below 2^-127, where those terms are below FP32 resolution against the
// others), products with the reference Hessian R = Hm 2^g carry 2^(g + E - F)
// (with the delta) or 2^(g - F) (with the orbit).  A diffabs(P, d) is taken
// only when its branch is known: P = 0 (|d|, with the reference's derivative
// convention sgn(0) = +1), or |d| < |P| / 2 (sgn(P) d); otherwise, and at
// orbit points that are both 0 or outside [2^-60, 2^40], the step runs in fr.
// The rounding is FP32's as in fr (one rounding per operation, FMAs where the
// compiler contracts), so the two forms agree to FP32 rounding.
// ---------------------------------------------------------------------------
struct BSFrame {
    float ux, uy; int E;          // deltas
    float s;                      // 2^E, 0 below 2^-127
    float cux, cuy;               // (a, b) 2^-E
    float h[4]; int F;            // Hessian, F = FR_ZERO_E when h = 0
    float am, bm; int ae, be;     // (a, b) = (am 2^ae, bm 2^be)
};

// 2^k for k clamped to [-127, 127] (2^-127 reads as 0)
FSG_DEV float fr_p2c(int k) { return __int_as_float((min(max(k, -127), 127) + 127) << 23); }
// unbiased exponent of |m| for a normal float, -127 for 0 and subnormals
FSG_DEV int fr_fexp(float m) { return ((__float_as_int(m) >> 23) & 0xff) - 127; }

FSG_DEV void frame_set_scale(BSFrame &S) {
    S.s = fr_p2c(S.E);
    S.cux = S.am * fr_p2c(S.ae - S.E);
    S.cuy = S.bm * fr_p2c(S.be - S.E);
}
FSG_DEV int frame_ec(const BSFrame &S) { return max(S.ae, S.be); }

// fr values -> frame (E >= the exponent of c minus 100, so that (a, b) 2^-E
// stays finite)
FSG_DEV void frame_in(BSFrame &S, fr xn, fr yn, const fr h[4]) {
    S.E = max(max(xn.e, yn.e), frame_ec(S) - 100);
    S.ux = xn.m * fr_p2c(xn.e - S.E);
    S.uy = yn.m * fr_p2c(yn.e - S.E);
    frame_set_scale(S);
    S.F = max(max(h[0].e, h[1].e), max(h[2].e, h[3].e));
    for (int k = 0; k < 4; k++) S.h[k] = h[k].m * fr_p2c(h[k].e - S.F);
}
FSG_DEV void frame_out(const BSFrame &S, fr &xn, fr &yn, fr h[4]) {
    xn = fr_norm(S.ux, S.E);
    yn = fr_norm(S.uy, S.E);
    for (int k = 0; k < 4; k++) h[k] = fr_norm(S.h[k], S.F);
}
// lazy renormalisation: max(|ux|, |uy|) and max |h| kept in [2^-30, 2^30]
FSG_DEV void frame_renorm(BSFrame &S) {
    const float m = fmaxf(fabsf(S.ux), fabsf(S.uy));
    if (!(m >= 0x1p-30f && m <= 0x1p30f)) {
        int En;
        if (m < 0x1p-126f) { S.ux = 0.f; S.uy = 0.f; En = frame_ec(S); }
        else {
            En = max(S.E + fr_fexp(m), frame_ec(S) - 100);
            const float sc = fr_p2c(S.E - En);
            S.ux *= sc; S.uy *= sc;
        }
        S.E = En;
        frame_set_scale(S);
    }
    const float mh = fmaxf(fmaxf(fabsf(S.h[0]), fabsf(S.h[1])),
                           fmaxf(fabsf(S.h[2]), fabsf(S.h[3])));
    if (!(mh >= 0x1p-30f && mh <= 0x1p30f)) {
        if (mh < 0x1p-126f) {
            for (int k = 0; k < 4; k++) S.h[k] = 0.f;
            S.F = FR_ZERO_E;
        } else {
            const int k = fr_fexp(mh);
            const float sc = fr_p2c(-k);
            for (int j = 0; j < 4; j++) S.h[j] *= sc;
            S.F += k;
        }
    }
}
// raise the Hessian's exponent to Fn (> F): entries below 2^(Fn - 127) drop
FSG_DEV void frame_raise_F(BSFrame &S, int Fn) {
    const float sc = fr_p2c(S.F - Fn);
    for (int k = 0; k < 4; k++) S.h[k] *= sc;
    S.F = Fn;
}
// h += Hm 2^g (the rebase's addition of the reference Hessian)
FSG_DEV void frame_add_hess(BSFrame &S, float4 Hm, int g) {
    if (Hm.x == 0.f && Hm.y == 0.f && Hm.z == 0.f && Hm.w == 0.f) return;
    if (g - S.F > 60) frame_raise_F(S, g - 30);
    const float k0 = fr_p2c(g - S.F);
    S.h[0] = fmaf(Hm.x, k0, S.h[0]); S.h[1] = fmaf(Hm.y, k0, S.h[1]);
    S.h[2] = fmaf(Hm.z, k0, S.h[2]); S.h[3] = fmaf(Hm.w, k0, S.h[3]);
}

// diffabs(P, d) for d = du 2^E and P known by its sign sp (0 when P = 0) and
// exponent bounds 2^elo <= |P| < 2^(ehi + 1) (burning_ship.py:19-60):
//   P = 0: |d| (with ddiffabsdX = -2 for d < 0, sgn(0) = +1);
//   |d| < |P| / 2: sgn(P) d;
//   |d| > 2^26 |P|: the sign of P + d is d's and 2 P is below FP32 resolution
//   against d.
// Returns false when the exponents leave the branch open.
FSG_DEV bool frame_diffabs(float sp, int elo, int ehi, float du, int E, float &val, float &dX,
                           float &dx) {
    const bool neg = du < 0.f;
    if (sp == 0.f) {
        val = neg ? -du : du; dX = neg ? -2.f : 0.f; dx = neg ? -1.f : 1.f;
        return true;
    }
    const float ad = fabsf(du);
    const int ed = ad == 0.f ? FR_ZERO_E : E + fr_fexp(ad);
    if (ed <= elo - 2) { val = sp * du; dX = 0.f; dx = sp; return true; }
    if (ed < ehi + 27) return false;
    if (sp > 0.f) { val = neg ? -du : du; dX = neg ? -2.f : 0.f; dx = neg ? -1.f : 1.f; }
    else { val = neg ? -du : du; dX = neg ? 0.f : 2.f; dx = neg ? -1.f : 1.f; }
    return true;
}
FSG_DEV float frame_sgn(float v, int e) {           // 0 for an exact 0
    return e == FR_ZERO_E ? 0.f : (signbit(v) ? -1.f : 1.f);
}

// One step of the loop at orbit point (X, Y) with the reference Hessian
// Hm 2^g (zero_ref: the zeros the loop uses right after a dynamic rebase),
// before renormalisation.  Returns false, leaving S untouched, when the step
// has to run in fr.
// DEEP: s = 0 (the deltas below 2^-127), where every product of two deltas,
// or of a delta and the Hessian, is 0 in the frame: those terms are left out.
template <bool DEEP>
FSG_DEV bool bs_frame_step(int flavor, bool hess, BSFrame &S, float X, float Y, int eX, int eY,
                           float4 Hm, int g, bool zero_ref) {
    const float s = DEEP ? 0.f : S.s, ux = S.ux, uy = S.uy;
    const float xs = DEEP ? 0.f : ux * s, ys = DEEP ? 0.f : uy * s;   // xn, yn as floats
    const float xx2 = ux * (DEEP ? 2.f * X : xs + 2.f * X);           // xn (xn + 2 X)
    const float yy2 = uy * (DEEP ? 2.f * Y : ys + 2.f * Y);           // yn (yn + 2 Y)
    const float xy = DEEP ? 0.f : ux * ys;                            // xn yn
    float v1 = 0.f, dX1 = 0.f, dx1 = 0.f, v2 = 0.f, dX2 = 0.f, dx2 = 0.f;
    float vy = 0.f, dXy = 0.f, dxy = 0.f;
    const bool use1 = flavor == 1 || flavor == 5, use2 = flavor >= 4;
    const bool usey = flavor == 2 || flavor == 3;
    const float sX = frame_sgn(X, eX), sY = frame_sgn(Y, eY);
    if (use1) {
        // P1 = X Y: 2^(eX + eY) <= |P1| < 2^(eX + eY + 2)
        // xn yn + xn Y + yn X
        const float o1 = DEEP ? fmaf(uy, X, ux * Y) : fmaf(uy, X, fmaf(ux, Y, xy));
        if (!frame_diffabs(sX * sY, eX + eY, eX + eY + 1, o1, S.E, v1, dX1, dx1)) return false;
    }
    if (use2) {
        // P2 = X^2 - Y^2 in the rounding of the fr closure (a component
        // below 2^-100 against one above 2^-60 drops out of it)
        const float P2 = __fsub_rn(__fmul_rn(X, X), __fmul_rn(Y, Y));
        const int e2 = fr_fexp(fabsf(P2));
        if (!frame_diffabs(P2 == 0.f ? 0.f : (P2 > 0.f ? 1.f : -1.f), e2, e2, xx2 - yy2, S.E,
                           v2, dX2, dx2))
            return false;
    }
    if (usey) {
        if (!frame_diffabs(sY, eY, eY, uy, S.E, vy, dXy, dxy)) return false;
    }
    // |Y + yn| and sgn(Y + yn) with sgn(0) = +1 (flavors 2, 3): the branch
    // is known here, so the sign is sgn(Y) unless |yn| dominates or Y = 0
    const float ab = DEEP ? fabsf(Y) : fabsf(Y + ys);
    const float sg = (sY != 0.f && dXy == 0.f) ? sY : (uy < 0.f ? -1.f : 1.f);
    if (hess) {
        const bool hz = zero_ref || (Hm.x == 0.f && Hm.y == 0.f && Hm.z == 0.f && Hm.w == 0.f);
        float k1 = 0.f, k0 = 0.f;
        if (!hz) {
            // the terms in 2^(g - F) are products with X or Y
            const bool need0 = (dX1 != 0.f || dX2 != 0.f || dXy != 0.f) && (X != 0.f || Y != 0.f);
            if (g + S.E - S.F > 60) frame_raise_F(S, g + S.E - 30);
            if (need0 && g - S.F > 60) frame_raise_F(S, g - 30);
            k1 = fr_p2c(g + S.E - S.F);
            k0 = need0 ? fr_p2c(g - S.F) : 0.f;
        } else {
            Hm = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const float h0 = S.h[0], h1 = S.h[1], h2 = S.h[2], h3 = S.h[3];
        float nxa, nxb, nya, nyb;
        if (DEEP) {
            // the same closures without the terms in s (xn = yn = 0 against X, Y)
            if (flavor == 1 || flavor == 2) {
                nxa = 2.f * (X * h0 + Hm.x * ux * k1) - 2.f * (Y * h2 + Hm.z * uy * k1);
                nxb = 2.f * (X * h1 + Hm.y * ux * k1) - 2.f * (Y * h3 + Hm.w * uy * k1);
            } else if (flavor == 3) {
                nxa = h0 * (2.f * X) + ux * (2.f * Hm.x * k1) - Hm.z * vy * k1
                      - Y * (Hm.z * dXy * k0 + h2 * dxy) - h2 * ab - sg * (uy * Hm.z * k1);
                nxb = h1 * (2.f * X) + ux * (2.f * Hm.y * k1) - Hm.w * vy * k1
                      - Y * (Hm.w * dXy * k0 + h3 * dxy) - h3 * ab - sg * (uy * Hm.w * k1);
            } else {
                const float dxa2 = h0 * (2.f * X) + ux * (2.f * Hm.x * k1)
                                   - h2 * (2.f * Y) - uy * (2.f * Hm.z * k1);
                const float dxb2 = h1 * (2.f * X) + ux * (2.f * Hm.y * k1)
                                   - h3 * (2.f * Y) - uy * (2.f * Hm.w * k1);
                const float dXa2 = 2.f * (X * Hm.x - Y * Hm.z) * k0;
                const float dXb2 = 2.f * (X * Hm.y - Y * Hm.w) * k0;
                nxa = dX2 * dXa2 + dx2 * dxa2;
                nxb = dX2 * dXb2 + dx2 * dxb2;
            }
            if (flavor == 1 || flavor == 5) {
                const float dxa = h0 * Y + h2 * X + (ux * Hm.z + uy * Hm.x) * k1;
                const float dxb = h1 * Y + h3 * X + (ux * Hm.w + uy * Hm.y) * k1;
                const float dXa = (Hm.x * Y + X * Hm.z) * k0, dXb = (Hm.y * Y + X * Hm.w) * k0;
                nya = 2.f * (dX1 * dXa + dx1 * dxa);
                nyb = 2.f * (dX1 * dXb + dx1 * dxb);
            } else if (flavor == 2) {
                nya = 2.f * (Hm.x * vy * k1 + X * (dXy * Hm.z * k0 + dxy * h2) + h0 * ab
                             + sg * (ux * Hm.z * k1));
                nyb = 2.f * (Hm.y * vy * k1 + X * (dXy * Hm.w * k0 + dxy * h3) + h1 * ab
                             + sg * (ux * Hm.w * k1));
            } else {
                nya = 2.f * ((Hm.x * uy + Hm.z * ux) * k1 + X * h2 + Y * h0);
                nyb = 2.f * ((Hm.y * uy + Hm.w * ux) * k1 + X * h3 + Y * h1);
            }
        } else if (flavor == 1 || flavor == 2) {
            nxa = 2.f * ((X + xs) * h0 + Hm.x * ux * k1) - 2.f * ((Y + ys) * h2 + Hm.z * uy * k1);
            nxb = 2.f * ((X + xs) * h1 + Hm.y * ux * k1) - 2.f * ((Y + ys) * h3 + Hm.w * uy * k1);
        } else if (flavor == 3) {
            nxa = h0 * (xs + 2.f * X) + ux * (h0 * s + 2.f * Hm.x * k1) - Hm.z * vy * k1
                  - Y * (Hm.z * dXy * k0 + h2 * dxy) - h2 * ab
                  - sg * (uy * Hm.z * k1 + uy * h2 * s);
            nxb = h1 * (xs + 2.f * X) + ux * (h1 * s + 2.f * Hm.y * k1) - Hm.w * vy * k1
                  - Y * (Hm.w * dXy * k0 + h3 * dxy) - h3 * ab
                  - sg * (uy * Hm.w * k1 + uy * h3 * s);
        } else {
            const float dxa2 = h0 * (xs + 2.f * X) + ux * (h0 * s + 2.f * Hm.x * k1)
                               - h2 * (ys + 2.f * Y) - uy * (h2 * s + 2.f * Hm.z * k1);
            const float dxb2 = h1 * (xs + 2.f * X) + ux * (h1 * s + 2.f * Hm.y * k1)
                               - h3 * (ys + 2.f * Y) - uy * (h3 * s + 2.f * Hm.w * k1);
            const float dXa2 = 2.f * (X * Hm.x - Y * Hm.z) * k0;
            const float dXb2 = 2.f * (X * Hm.y - Y * Hm.w) * k0;
            nxa = dX2 * dXa2 + dx2 * dxa2;
            nxb = dX2 * dXb2 + dx2 * dxb2;
        }
        if (DEEP) {
        } else if (flavor == 1 || flavor == 5) {
            const float dxa = (h0 * uy + ux * h2) * s + h0 * Y + h2 * X
                              + (ux * Hm.z + uy * Hm.x) * k1;
            const float dxb = (h1 * uy + ux * h3) * s + h1 * Y + h3 * X
                              + (ux * Hm.w + uy * Hm.y) * k1;
            const float dXa = (Hm.x * Y + X * Hm.z) * k0, dXb = (Hm.y * Y + X * Hm.w) * k0;
            nya = 2.f * (dX1 * dXa + dx1 * dxa);
            nyb = 2.f * (dX1 * dXb + dx1 * dxb);
        } else if (flavor == 2) {
            nya = 2.f * (Hm.x * vy * k1 + X * (dXy * Hm.z * k0 + dxy * h2) + h0 * ab
                         + sg * (ux * Hm.z * k1 + ux * h2 * s));
            nyb = 2.f * (Hm.y * vy * k1 + X * (dXy * Hm.w * k0 + dxy * h3) + h1 * ab
                         + sg * (ux * Hm.w * k1 + ux * h3 * s));
        } else {
            nya = 2.f * ((Hm.x * uy + Hm.z * ux) * k1 + X * h2 + Y * h0 + (h0 * uy + ux * h2) * s);
            nyb = 2.f * ((Hm.y * uy + Hm.w * ux) * k1 + X * h3 + Y * h1 + (h1 * uy + ux * h3) * s);
        }
        S.h[0] = nxa; S.h[1] = nxb; S.h[2] = nya; S.h[3] = nyb;
    }
    float nx, ny;
    if (flavor == 1) {
        nx = xx2 - yy2 + S.cux; ny = 2.f * v1 - S.cuy;
    } else if (flavor == 2) {
        nx = xx2 - yy2 + S.cux; ny = 2.f * (X * vy + ux * ab) - S.cuy;
    } else if (flavor == 3) {
        nx = xx2 - Y * vy - uy * ab + S.cux;
        ny = 2.f * (DEEP ? X * uy + Y * ux : X * uy + Y * ux + xy) - S.cuy;
    } else if (flavor == 4) {
        nx = v2 + S.cux; ny = 2.f * (DEEP ? X * uy + Y * ux : X * uy + Y * ux + xy) - S.cuy;
    } else {
        nx = v2 + S.cux; ny = 2.f * v1 - S.cuy;
    }
    S.ux = nx; S.uy = ny;
    return true;
}

// The step at an orbit point X = Y = 0 (every term is a product of two deltas
// or c): the deltas' exponent moves to E' = max(2 E, Ec - 100) and the
// Hessian's to F + E' - E, so that the general step's products "u u s" and
// "h u s" with s = 2^(2E - E') land in the new frames (its products with X
// and Y vanish).
FSG_DEV void bs_frame_step_zero(int flavor, bool hess, BSFrame &S, float4 Hm, int g,
                                bool zero_ref) {
    const int E = S.E;
    const int En = max(2 * E, frame_ec(S) - 100);
    BSFrame T = S;
    T.s = fr_p2c(2 * E - En);
    T.cux = S.am * fr_p2c(S.ae - En);
    T.cuy = S.bm * fr_p2c(S.be - En);
    if (T.F != FR_ZERO_E) T.F = S.F + En - E;
    // all diffabs arguments are 0 here: the step is always taken
    bs_frame_step<false>(flavor, hess, T, 0.f, 0.f, FR_ZERO_E, FR_ZERO_E, Hm, g, zero_ref);
    S = T;
    S.E = En;
    frame_set_scale(S);
}

// bs_frame_step for flavor 1 where the orbit is real (Y = 0 and Hm.y = Hm.z = 0 at
// every point): the fold's argument is 0 at the orbit, so its branch is the sign
// of the change, and the terms with zeros are left out.  The roundings are those
// of the general form's contracted sums with those terms 0 (spelled out where a
// shorter sum would contract otherwise).
template <bool DEEP>
FSG_DEV void bs_frame_step_axis1(bool hess, BSFrame &S, float X, float Y, float4 Hm, int g,
                                 bool zero_ref) {
    const float s = DEEP ? 0.f : S.s, ux = S.ux, uy = S.uy;
    const float xs = DEEP ? 0.f : ux * s, ys = DEEP ? 0.f : uy * s;
    const float xx2 = ux * (DEEP ? 2.f * X : xs + 2.f * X);
    const float yy2 = uy * (DEEP ? 2.f * Y : ys + 2.f * Y);
    const float o1 = DEEP ? __fmul_rn(uy, X) : fmaf(uy, X, __fmul_rn(ux, ys));
    const bool neg = o1 < 0.f;
    const float v1 = neg ? -o1 : o1, dx1 = neg ? -1.f : 1.f;
    if (hess) {
        const bool hz = zero_ref || (Hm.x == 0.f && Hm.w == 0.f);
        float k1 = 0.f, dXb = 0.f;
        if (!hz) {
            const bool need0 = neg && X != 0.f;
            if (g + S.E - S.F > 60) frame_raise_F(S, g + S.E - 30);
            if (need0) {
                if (g - S.F > 60) frame_raise_F(S, g - 30);
                dXb = __fmul_rn(__fmul_rn(X, Hm.w), fr_p2c(g - S.F));
            }
            k1 = fr_p2c(g + S.E - S.F);
        } else {
            Hm = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const float h0 = S.h[0], h1 = S.h[1], h2 = S.h[2], h3 = S.h[3];
        float nxa, nxb, dxa, dxb;
        if (DEEP) {
            nxa = 2.f * (X * h0 + Hm.x * ux * k1) - 2.f * (Y * h2);
            nxb = 2.f * (X * h1) - 2.f * (Y * h3 + Hm.w * uy * k1);
            dxa = fmaf(__fmul_rn(uy, Hm.x), k1, __fmul_rn(h2, X));
            dxb = fmaf(__fmul_rn(ux, Hm.w), k1, __fmul_rn(h3, X));
        } else {
            nxa = 2.f * ((X + xs) * h0 + Hm.x * ux * k1) - 2.f * __fmul_rn(Y + ys, h2);
            nxb = 2.f * __fmul_rn(X + xs, h1) - 2.f * ((Y + ys) * h3 + Hm.w * uy * k1);
            dxa = fmaf(__fmul_rn(uy, Hm.x), k1, fmaf(h2, X, __fmul_rn(h0 * uy + ux * h2, s)));
            dxb = fmaf(__fmul_rn(ux, Hm.w), k1, fmaf(h3, X, __fmul_rn(h1 * uy + ux * h3, s)));
        }
        S.h[0] = nxa; S.h[1] = nxb;
        S.h[2] = 2.f * (dx1 * dxa);
        S.h[3] = neg ? 2.f * fmaf(-2.f, dXb, -dxb) : 2.f * dxb;
    }
    S.ux = xx2 - yy2 + S.cux;
    S.uy = 2.f * v1 - S.cuy;
}

// bs_frame_step_zero for flavor 1 right after a rebase (the reference Hessian
// reads as 0): products of deltas and c alone.
FSG_DEV void bs_frame_zero1(bool hess, BSFrame &S) {
    const int E = S.E;
    const int En = max(2 * E, frame_ec(S) - 100);
    const float s = fr_p2c(2 * E - En), ux = S.ux, uy = S.uy;
    const float xs = ux * s, ys = uy * s;
    const float xy = __fmul_rn(ux, ys);
    const bool neg = xy < 0.f;
    if (hess) {
        const float h0 = S.h[0], h1 = S.h[1], h2 = S.h[2], h3 = S.h[3];
        const float dxa = __fmul_rn(h0 * uy + ux * h2, s), dxb = __fmul_rn(h1 * uy + ux * h3, s);
        S.h[0] = 2.f * __fmul_rn(xs, h0) - 2.f * __fmul_rn(ys, h2);
        S.h[1] = 2.f * __fmul_rn(xs, h1) - 2.f * __fmul_rn(ys, h3);
        S.h[2] = neg ? -2.f * dxa : 2.f * dxa;
        S.h[3] = neg ? -2.f * dxb : 2.f * dxb;
    }
    if (S.F != FR_ZERO_E) S.F += En - E;
    S.E = En;
    frame_set_scale(S);
    S.ux = ux * xs - uy * ys + S.cux;
    S.uy = 2.f * (neg ? -xy : xy) - S.cuy;
}

// |X + d| <= |d| for one component (d = du 2^E), as the fr values round:
// true when X = 0 or |X| < 2^-25 |d| (X + d rounds to d), false when
// |d| < |X| / 2; open otherwise
FSG_DEV bool frame_le(float du, int E, int eX, bool &le) {
    if (eX == FR_ZERO_E) { le = true; return true; }
    const float ad = fabsf(du);
    const int ed = ad == 0.f ? FR_ZERO_E : E + fr_fexp(ad);
    if (ed <= eX - 2) { le = false; return true; }
    if (ed >= eX + 26) { le = true; return true; }
    return false;
}
// The loop's tests at orbit point (X, Y) (perturbation.py:1627-1711) in the
// frame form: 0 none, 1 escape, 2 rebase where X + xn, Y + yn round to xn, yn
// (the deltas stay), 3 to be decided in fr
FSG_DEV int bs_frame_tests(const BSFrame &S, float X, float Y, int eX, int eY, float M2s,
                           bool div_rebase) {
    bool lex, ley;
    if (S.E > 10) return 3;                             // deltas above 2^40: fr from here
    if (!frame_le(S.ux, S.E, eX, lex) || !frame_le(S.uy, S.E, eY, ley)) return 3;
    const float XX = fmaf(S.ux, S.s, X), YY = fmaf(S.uy, S.s, Y);
    const float q = fmaf(XX, XX, YY * YY);
    if (fabsf(q - M2s) <= M2s * 0x1p-18f) return 3;
    if (q > M2s) return 1;
    if (div_rebase || (lex && ley)) return (lex && ley) ? 2 : 3;
    return 0;
}

// One step of flavor 1 in the double form, bs_hess and bs_zn with their products
// on the integer pipes: false (nothing changed) where one of them is left open.
// xs = X + xn, ys = Y + yn.  The FP64 pipe sees 24 sums instead of the 69
// instructions of the plain form: what belongs to the fold's other branch (the
// reference's own d(XY), with ddiffabsdX = 0) is taken only there.
// AXIS: the orbit is real (Y = Xb = Ya = 0 at every point: the nuclei that a
// Newton search from the ship's antenna finds).  A third of the products are then
// zeros, and a sum with a zero is its other term while that is not 0: they are
// left out, for 15 sums, and a result that comes out as 0, whose sign they could
// change, refuses the step.
template <bool AXIS>
FSG_DEV bool bs_step_ship(bool hess, double &xn, double &yn, double h[4], double X, double Y, double xs,
                          double ys, double Xa, double Xb, double Ya, double Yb, double a, double b) {
    bool ok = true;
    double x2 = xn;                              // xn + 2 X (X = 0 once per rebase)
    if (!d_is0(X) | d_is0(xn)) x2 = d_add_here(xn, d_twice(X));
    const sfac fx = sfac_of(xn), fy = sfac_of(yn), fX = sfac_of(X), fY = sfac_of(Y);
    // the fold |X Y|: opx its argument's change, `first` its sign at the orbit,
    // `same` whether the argument keeps it, s1 = ddiffabsdx
    double opX = 0., opx = sfac_mul(fx, fy, ok);
    bool first = true, same;
    if (AXIS) {
        opx += sfac_mul(fy, fX, ok);
        ok &= !d_is0(opx) & !d_is0(yn);
        same = d_ge0(opx);
    } else {
        opx = opx + sfac_mul(fx, fY, ok) + sfac_mul(fy, fX, ok);
        opX = sfac_mul(fX, fY, ok);
        const double t = opX + opx;
        first = d_ge0(opX);
        same = first ? d_ge0(t) : d_le0(t);
    }
    const unsigned s1 = first == same ? 0u : 0x80000000u;
    double fold = opx;
    if (!AXIS && !same) fold = d_add_here(d_twice(opX), opx);
    const double y2 = AXIS ? yn : yn + d_twice(Y);
    const double nx = sfac_mul(fx, sfac_of(x2), ok) - sfac_mul(fy, AXIS ? fy : sfac_of(y2), ok) + a;
    const double ny = d_twice(d_flip(fold, s1)) - b;
    if (hess) {
        const sfac xa = sfac_of(h[0]), xb = sfac_of(h[1]), ya = sfac_of(h[2]), yb = sfac_of(h[3]);
        const sfac fXa = sfac_of(Xa), fYb = sfac_of(Yb), fs = sfac_of(xs);
        double da = sfac_mul(xa, fy, ok) + sfac_mul(fx, ya, ok);
        double db = sfac_mul(xb, fy, ok) + sfac_mul(fx, yb, ok);
        double nxa = sfac_mul(fs, xa, ok) + sfac_mul(fXa, fx, ok), nxb = sfac_mul(fs, xb, ok);
        double va, vb;
        if (AXIS) {
            da = da + sfac_mul(ya, fX, ok) + sfac_mul(fy, fXa, ok);
            db = db + sfac_mul(fx, fYb, ok) + sfac_mul(yb, fX, ok);
            va = sfac_mul(fy, ya, ok);
            vb = sfac_mul(fy, yb, ok) + sfac_mul(fYb, fy, ok);
        } else {
            const sfac fXb = sfac_of(Xb), fYa = sfac_of(Ya), ft = sfac_of(ys);
            da = da + sfac_mul(xa, fY, ok) + sfac_mul(fx, fYa, ok) + sfac_mul(ya, fX, ok) + sfac_mul(fy, fXa, ok);
            db = db + sfac_mul(xb, fY, ok) + sfac_mul(fx, fYb, ok) + sfac_mul(yb, fX, ok) + sfac_mul(fy, fXb, ok);
            nxb += sfac_mul(fXb, fx, ok);
            va = sfac_mul(ft, ya, ok) + sfac_mul(fYa, fy, ok);
            vb = sfac_mul(ft, yb, ok) + sfac_mul(fYb, fy, ok);
        }
        ok &= !(d_is0(da) | d_is0(db));
        if (!same) {
            // ddiffabsdX = 2 s1 times the reference's d(XY)
            double dXb = d_mul_here(X, Yb);
            if (!AXIS) {
                dXb = d_add_here(d_mul_here(Xb, Y), dXb);
                da = d_add_here(d_twice(d_add_here(d_mul_here(Xa, Y), d_mul_here(X, Ya))), da);
            }
            db = d_add_here(d_twice(dXb), db);
        }
        nxa = d_twice(nxa) - d_twice(va);
        nxb = d_twice(nxb) - d_twice(vb);
        if (AXIS) ok &= !(d_is0(db) | d_is0(nxa) | d_is0(nxb));
        if (!ok) return false;
        h[0] = nxa; h[1] = nxb; h[2] = d_twice(d_flip(da, s1)); h[3] = d_twice(d_flip(db, s1));
    }
    if (!ok) return false;
    xn = nx; yn = ny;
    return true;
}

// a1 b1 + a2 b2 (minus: a1 b1 - a2 b2): 58 binary orders apart only the larger
// product is taken
FSG_DEV double d_two_far(double a1, double b1, double a2, double b2, bool minus) {
    const int e1 = d_field(a1) + d_field(b1), e2 = d_field(a2) + d_field(b2);
    const unsigned flip = minus ? 0x80000000u : 0u;
    if (abs(e1 - e2) >= 59 && max(e1, e2) >= 1025) {
        const bool first = e1 > e2;
        return d_mul_here(first ? a1 : d_flip(a2, flip), first ? b1 : b2);
    }
    return d_add_far(d_mul_here(a1, b1), d_flip(d_mul_here(a2, b2), flip));
}

// the exponent field of x, continued below 1 for subnormals, far below any for 0
FSG_DEV int d_field0(double x) {
    const int f = d_field(x);
    if (f != 0) return f;
    return d_is0(x) ? -20000 : 12 - __clzll((long long)(dbits(x) << 1 >> 1));
}
// signs of products as words whose top bit counts
FSG_DEV unsigned d_sgn2(double a, double b) { return d_hi(a) ^ d_hi(b); }
FSG_DEV double d_zero_of(unsigned s) { return d_zero((s >> 31) != 0u); }

// The same step at X = Y = +0 right after a rebase (the reference Hessian reads
// as 0): products of deltas and c alone.  The plain form's other terms are zeros:
// beside a sum that is not 0 they change nothing, and a sum of da or db that is 0
// comes out as +0 whatever their signs (xa yn, xa 0 and yn 0 are not all negative).
FSG_DEV bool bs_ship_crit(bool hess, double &xn, double &yn, double h[4], double a, double b) {
    const int x = d_field(xn), y = d_field(yn);
    if (max(x, y) > 1023 - 58 || min(x, y) == 0) return false;
    // the fold's sign, its value only where it takes part in the sum with b
    unsigned s1 = (d_hi(xn) ^ d_hi(yn)) & 0x80000000u;
    double nx = a, ny = d_flip(b, 0x80000000u);
    if (d_field(b) + 1023 - x - y < 59 || x + y < 1025) {
        const double op = d_mul_here(xn, yn);
        if (d_is0(op)) s1 = 0u;
        ny = d_add_far(d_twice(d_flip(op, s1)), ny);
    }
    if (d_field(a) + 1023 - 2 * max(x, y) < 59) nx = d_add_far(d_two_far(xn, xn, yn, yn, true), a);
    if (hess) {
        const double xa = h[0], xb = h[1], ya = h[2], yb = h[3];
        const int top = max(max(d_field0(xa), d_field0(xb)), max(d_field0(ya), d_field0(yb)));
        if (top > 1900) return false;            // (infinities and NaN times a zero)
        double da = 0., db = 0., na, nb;
        if (max(x, y) + top <= 968) {
            // every product underflows: the zeros' signs
            na = d_zero_of(d_sgn2(xn, xa) & d_hi(xn) & ~(d_sgn2(yn, ya) & d_hi(yn)));
            nb = d_zero_of(d_sgn2(xn, xb) & d_hi(xn) & ~(d_sgn2(yn, yb) & d_hi(yn)));
        } else {
            da = d_two_far(xa, yn, xn, ya, false);
            db = d_two_far(xb, yn, xn, yb, false);
            na = d_two_far(xn, xa, yn, ya, true);
            nb = d_two_far(xn, xb, yn, yb, true);
            if (d_is0(da)) da = 0.;
            if (d_is0(db)) db = 0.;
            if (d_is0(na) | d_is0(nb)) return false;
        }
        h[0] = d_twice(na);
        h[1] = d_twice(nb);
        h[2] = d_twice(d_flip(da, s1));
        h[3] = d_twice(d_flip(db, s1));
    }
    xn = nx; yn = ny;
    return true;
}

// bs_step_ship on the real axis far below the orbit (views whose deltas are 58
// binary orders under X): products of two deltas are below half an ulp of the sum
// that they enter, so neither they nor the sums are taken.  Exponent fields say
// so for each sum (a product's exponent is the sum of its factors', or one more;
// `far` binary orders leave a power of two its ulp): 10 products and 6 sums
// remain of 18 and 15.  The integer pipes take four of the products: 255^2 pixels
// of the period-12 nucleus to 20000 iterations take 35.7 ms with four or six of
// them there, 37.2 with two, 39.3 with none, 67 without this step and
// bs_ship_crit.  Yz, Xb, Ya: zeros, for the signs of results that are 0
// because all their terms are.  false (nothing changed) where a sum is open.
FSG_DEV bool bs_ship_deep(bool hess, double &xn, double &yn, double h[4], double X, double Yz, double Xa,
                          double Xb, double Ya, double Yb, double a, double b) {
    const int far = 55;
    const int x = d_field(xn), y = d_field(yn), fX = d_field(X);
    // (everything that the factors' fields can tell is settled ahead of the
    // products: an integer test waits 100 clocks for an FP64 result)
    bool ok = (fX - max(x, y) >= far + 3) & (min(x, y) >= 1) & (min(x, y) + fX >= 1025)
              & (x + fX >= 2 * y + 2 + far);                 // yn yn beside xn (xn + 2 X)
    const unsigned s1 = d_sgn2(yn, X) & 0x80000000u;
    if (!ok) return false;
    const dfac dX = dfac_of(X);
    dfac dX2 = dX;
    dX2.s += 0x00100000u;
    const double px = dfac_mul(dfac_of(xn), dX2, ok), op = dfac_mul(dfac_of(yn), dX, ok);
    double n0 = 0., n1 = 0., n2 = 0., n3 = 0.;
    if (hess) {
        // exponents of da = ((xa yn + xn ya) + ya X) + yn Xa and of
        // db = ((xb yn + xn yb) + xn Yb) + yb X
        const double ha = h[0], hb = h[1], ga = h[2], gb = h[3];
        const int xa = d_field0(ha), xb = d_field0(hb), ya = d_field0(ga), yb = d_field0(gb);
        const int fXa = d_field(Xa), fYb = d_field(Yb);
        const int sa = max(xa + y, x + ya) + 2, ta = ya + fX, ua = y + fXa;
        const int sb = max(xb + y, x + yb) + 2, tb = x + fYb, ub = yb + fX;
        const bool a3 = ta - sa >= far, b3 = tb - sb >= far;
        ok &= (min(fXa, fYb) >= 1)
              & (max(max(max(xa, xb), max(ya, yb)), max(max(fXa, fYb), fX)) <= 1900);
        ok &= a3 | (ua - max(sa, ta + 2) >= far + 1);
        ok &= b3 | (ub - max(sb, tb + 2) >= far + 1);
        if (!ok) return false;
        n2 = d_mul_here(yn, Xa);
        double gx;
        if (min(ya, yb) + fX >= 1025) {
            gx = dfac_mul(dfac_of(ga), dX, ok);
            n3 = dfac_mul(dfac_of(gb), dX, ok);
            if (!ok) return false;
        } else {
            gx = d_mul_here(ga, X);
            n3 = d_mul_here(gb, X);
        }
        n0 = d_mul_here(Xa, xn);
        n1 = d_mul_here(Yb, yn);                 // vb = yn yb + Yb yn
        if (fYb - yb < far + 2) n1 = d_add_here(d_mul_here(yn, gb), n1);
        n1 = d_flip(d_twice(n1), 0x80000000u);
        if (a3) n2 = d_add_here(gx, n2);
        if (b3) n3 = d_add_here(d_mul_here(xn, Yb), n3);
        n0 = d_add_here(d_mul_here(X, ha), n0);
        n1 = d_add_here(d_twice(d_mul_here(X, hb)), n1);
        // va = yn ya
        if (!((d_field(n0) >= max(y + ya - 1023 + 2 + far, 1)) | (y + ya <= 968))) return false;
        n0 = d_twice(n0);
        if (s1) n3 = d_add_here(d_twice(d_mul_here(X, Yb)), n3);
        if (d_is0(n0) | d_is0(n1) | d_is0(n2) | d_is0(n3)) {
            // a sum whose terms all underflow has the sign that their zeros add to
            const bool x3 = d_is0(n3);
            const unsigned pa = d_sgn2(ha, yn) & d_sgn2(xn, ga) & d_sgn2(ha, Yz) & d_sgn2(xn, Ya)
                                & d_sgn2(ga, X) & d_sgn2(yn, Xa);
            const unsigned pb = d_sgn2(hb, yn) & d_sgn2(xn, gb) & d_sgn2(hb, Yz) & d_sgn2(xn, Yb)
                                & d_sgn2(gb, X) & d_sgn2(yn, Xb);
            const unsigned da = d_sgn2(Xa, Yz) & d_sgn2(X, Ya), db = d_sgn2(X, Yb);
            if (d_is0(n0)) {
                if (!(d_is0(d_mul_here(X, ha)) & d_is0(d_mul_here(Xa, xn)))) return false;
                n0 = d_zero_of(d_sgn2(X, ha) & d_sgn2(Xa, xn) & ~(d_sgn2(yn, ga) & d_sgn2(Ya, yn)));
            }
            if (d_is0(n1)) {
                if (!(d_is0(d_mul_here(X, hb)) & d_is0(d_mul_here(Yb, yn)) & d_is0(d_mul_here(yn, gb)))) return false;
                n1 = d_zero_of(d_sgn2(X, hb) & d_sgn2(Xb, xn) & ~(d_sgn2(yn, gb) & d_sgn2(Yb, yn)));
            }
            if (d_is0(n2)) {
                if (!(d_is0(d_mul_here(ga, X)) & d_is0(d_mul_here(yn, Xa)))) return false;
                // ddiffabsdX (0 or -2) times the reference's d(XY), and ddiffabsdx times this
                n2 = d_flip(d_zero_of(s1 ? ~da & ~pa : da & pa), s1);
            }
            if (x3) {
                if ((s1 != 0u) | !(d_is0(d_mul_here(gb, X)) & d_is0(d_mul_here(xn, Yb)))) return false;
                n3 = d_zero_of(db & pb);
            }
        }
        h[0] = n0; h[1] = n1; h[2] = d_twice(d_flip(n2, s1)); h[3] = d_twice(d_flip(n3, s1));
    }
    if (!ok) return false;
    xn = d_add_here(px, a);
    yn = d_add_here(d_twice(d_flip(op, s1)), d_flip(b, 0x80000000u));
    return true;
}

// a + b; flavor 1 in the double form looks whether there is a sum to take
template <class T, int FL> FSG_DEV T bs_add(T a, T b) { return a + b; }
template <> FSG_DEV double bs_add<double, 1>(double a, double b) { return d_add_far(a, b); }

template <class T> struct IsDouble { static constexpr bool value = false; };
template <> struct IsDouble<double> { static constexpr bool value = true; };
template <class T> struct IsFr { static constexpr bool value = false; };
template <> struct IsFr<fr> { static constexpr bool value = true; };
template <class T> struct IsXr { static constexpr bool value = false; };
template <> struct IsXr<xf> { static constexpr bool value = true; };

// FL: the flavor as a compile-time constant (1..5), or 0 to read C.flavor.  AXIS:
// every reference of the launch is real (RefDev.axis), flavor 1
template <class T, int FL, bool AXIS>
FSG_DEV int pixel_bs(const TileDev &T_, const CalcDev &C, long long ip, unsigned &nfull,
                     unsigned &nbla, unsigned &nreb) {
    const TileDev &Tl = T_;
    const RefDev &R = *Tl.ref;
    const long long np = (long long)Tl.nx * Tl.ny;
    const int flavor = FL ? FL : C.flavor;
    const bool hess = C.calc_dzndc != 0;
    const int order = R.order, div_iter = R.div_iter;
    // perturbation.py:2260-2280 ref_path_c_from_pix_BS through Xrange values
    double2 pp = fsg_pixel(Tl, ip);
    double px = pp.x, py = pp.y;
    double x1 = Tl.lin[0] * px + Tl.lin[1] * py;
    double y1 = Tl.lin[2] * px + Tl.lin[3] * py;
    xf dxr; dxr.m = Tl.dx_m; dxr.e = Tl.dx_e;
    xc c_xr = xf_mul_c(dxr, cx(x1, y1));
    double ar, br; int ae, be;
    xr_coexp_r(c_xr.re, c_xr.e, Tl.drift_re, Tl.drift_e, ar, br, ae);
    const T a = from_me<T>(ar + br, ae);
    xr_coexp_r(c_xr.im, c_xr.e, Tl.drifty_m, Tl.drifty_e, ar, br, be);
    const T b = from_me<T>(ar + br, be);

    T xn = cst<T>(0.f), yn = cst<T>(0.f);
    T h[4] = {cst<T>(0.f), cst<T>(0.f), cst<T>(0.f), cst<T>(0.f)};
    const fr M2f = fr_from_d(C.M2);
    int w = 0, n = 0; signed char stop = -1; bool dyn = true;
    // double form: X_w + xn and Y_w + yn of the last test, while they stand
    double XX_last = 0., YY_last = 0.; bool has_sums = false;
    // whether c is far enough below the orbit for bs_ship_crit and bs_ship_deep
    bool below = false;
    if constexpr (IsDouble<T>::value && FL == 1) {
        below = max(d_field(a), d_field(b)) <= 1023 - 58;
    }
    // calc_orbit snapshots (perturbation.py:1501-1508), the reference's two
    // forms only: the FP32 + exponent instantiation compiles without them
    constexpr bool FR_FORM = IsFr<T>::value;
    constexpr bool XR_FORM = IsXr<T>::value;
    constexpr bool ORB_FORM = !FR_FORM;
    const int bs = ORB_FORM ? C.backshift : 0;
    OrbitSnap<double2> S;
    S.init(bs, cx(0., 0.));
    // the reference's BLA step (perturbation.py:1520-1545, 1793-1811)
    auto apply_bla = [&](int step, int ib) {
        T M[8];
        BSRef<T>::bla(R, ib, M);
        n += step; w = (w + step) % order;
        T nx = M[0] * xn + M[1] * yn + M[4] * a + M[5] * b;
        T ny = M[2] * xn + M[3] * yn + M[6] * a + M[7] * b;
        xn = nx; yn = ny;
        if (hess) {
            T xa = M[0] * h[0] + M[1] * h[2], xb = M[0] * h[1] + M[1] * h[3];
            T ya = M[2] * h[0] + M[3] * h[2], yb = M[2] * h[1] + M[3] * h[3];
            h[0] = xa; h[1] = xb; h[2] = ya; h[3] = yb;
        }
        nbla++;
    };
    // frame form of the FP32 + exponent loop (BSFrame); the fr values are
    // current whenever frm is false
    BSFrame Fm;
    bool frm = false;
    float M2s = 0.f;
    // with |X|, |Y| and the deltas below 2^(eMlim + 1), |Z + dz|^2 < M2 / 8
    const int eMlim = min((M2f.e >> 1) - 4, 40);
    if constexpr (FR_FORM) {
        Fm.am = a.m; Fm.ae = a.e; Fm.bm = b.m; Fm.be = b.e;
        M2s = (float)C.M2;
    }
    for (;;) {
        bool bla_done = false, stepped = false;
        if constexpr (FR_FORM) {
            if (frm) {
            // Steps in the frame form from orbit point w on, until the loop ends
            // (0), a BLA step was taken (1), the step at w has to run in fr (2) or
            // the tests at w have to (3); the fr values are current on return.
            auto frame_run = [&]() -> int {
                // the records of w, read together as soon as w is known; flavor 5
                // reads the Hessian's where it uses it: its views leave the frame
                // form for fr steps often, and need it at fewer points (100^2
                // pixels of a period-17 nucleus to 3000 iterations: 8.80 ms with
                // all three, 8.50 so)
                constexpr bool HM_LATE = FL == 5;
                int4 fz;
                float4 fa, Hm = make_float4(0.f, 0.f, 0.f, 0.f);
                auto fetch = [&]() {
                    const int4 *at = R.bs_at + 3 * (size_t)w;
                    fz = __ldg(at);
                    fa = __ldg((const float4 *)at + 1);
                    if (hess && !HM_LATE) Hm = __ldg((const float4 *)at + 2);
                };
                auto fetch_late = [&]() {
                    if (hess) Hm = __ldg((const float4 *)(R.bs_at + 3 * (size_t)w) + 2);
                };
                fetch();
                const bool bla_on = C.bla && R.bla_len > 0;
                // X_0 = Y_0 = 0 and no BLA attempt there (the loop's own condition):
                // after a rebase the step at w = 0 follows at once.  200^2 pixels of
                // a period-12 nucleus to 3000 iterations: 1.41 ms, 1.61 without
                const bool crit0 = FL == 1 && (__ldg(&R.bs_at[0]).x & 4)
                                   && !(bla_on && (1 << FSG_STG_COMPRESSED) < R.first_invalid
                                        && bla_possible(R, 0));
                for (;;) {
                    if (bla_on && (w & 7) == 0 &&
                        (1 << FSG_STG_COMPRESSED) < R.first_invalid - w && bla_possible(R, w)) {
                        int ib;
                        const int step = BLAGet<T>::get(R, fr_norm(Fm.ux, Fm.E),
                                                        fr_norm(Fm.uy, Fm.E), w, ib);
                        if (step != 0) {
                            frame_out(Fm, xn, yn, h);
                            apply_bla(step, ib);
                            return 1;
                        }
                    }
                    if (!(fz.x & 5)) { frame_out(Fm, xn, yn, h); return 2; }
                    if constexpr (HM_LATE) {
                        if (dyn) Hm = make_float4(0.f, 0.f, 0.f, 0.f);
                        else fetch_late();
                    }
                    if (fz.x & 4) {
                        if (FL == 1 && dyn) bs_frame_zero1(hess, Fm);
                        else bs_frame_step_zero(flavor, hess, Fm, Hm, fz.y, dyn);
                    } else if (AXIS) {
                        if (Fm.s == 0.f) bs_frame_step_axis1<true>(hess, Fm, fa.x, fa.y, Hm, fz.y, dyn);
                        else bs_frame_step_axis1<false>(hess, Fm, fa.x, fa.y, Hm, fz.y, dyn);
                    } else {
                        const int eX = __float_as_int(fa.z), eY = __float_as_int(fa.w);
                        const bool ok = Fm.s == 0.f
                            ? bs_frame_step<true>(flavor, hess, Fm, fa.x, fa.y, eX, eY, Hm,
                                                  fz.y, dyn)
                            : bs_frame_step<false>(flavor, hess, Fm, fa.x, fa.y, eX, eY, Hm,
                                                   fz.y, dyn);
                        if (!ok) {
                            frame_out(Fm, xn, yn, h);
                            return 2;
                        }
                    }
                after_step:
                    w += 1;
                    if (w >= order) w = 0;                  // w < order before
                    fetch();
                    frame_renorm(Fm);
                    n += 1;
                    nfull++;
                    if (n >= C.max_iter) {
                        // (the step that reaches it leaves w where it was)
                        w = (w == 0 ? order : w) - 1;
                        stop = 0; frame_out(Fm, xn, yn, h); return 0;
                    }
                    // deltas below the orbit point's bound: no escape, no rebase
                    const int ed = Fm.E + fr_fexp(fmaxf(fabsf(Fm.ux), fabsf(Fm.uy)));
                    if (ed <= min(fz.z, eMlim) && fz.w <= eMlim) { dyn = false; continue; }
                    const bool divr = w >= div_iter - 1;
                    int res = 3;
                    if ((fz.x & 4) && ed <= eMlim && Fm.E <= 10) {
                        res = 2;               // X = Y = 0, no escape
                    } else if (fz.x & 2) {
                        res = bs_frame_tests(Fm, fa.x, fa.y, __float_as_int(fa.z),
                                             AXIS ? FR_ZERO_E : __float_as_int(fa.w), M2s, divr);
                    }
                    if (res == 0) { dyn = false; continue; }
                    if (res == 1) { stop = 1; frame_out(Fm, xn, yn, h); return 0; }
                    if (res == 2) {
                        // rebase where X + xn, Y + yn round to the deltas: they stay
                        if constexpr (HM_LATE) fetch_late();
                        if (hess) frame_add_hess(Fm, Hm, fz.y);
                        if (!divr) dyn = true;
                        const bool there = w == 0;
                        w = 0; nreb++;
                        if (FL == 1 && dyn && crit0) {
                            bs_frame_zero1(hess, Fm);
                            goto after_step;
                        }
                        if (!there) fetch();
                        continue;
                    }
                    frame_out(Fm, xn, yn, h);
                    return 3;
                }
            };
                frm = false;
                const int r = frame_run();
                if (r == 0) break;
                if (r == 1) continue;
                bla_done = true;
                stepped = r == 3;
            }
        }
        if (!stepped) {
            if (C.bla && R.bla_len > 0 && !bla_done && (w & 7) == 0) {
                int ib;
                // the reference compares the double value of |dz| (0 when it
                // underflows, perturbation.py:1123-1135)
                const int step = BLAGet<T>::get(R, xn, yn, w, ib);
                if (step != 0) { apply_bla(step, ib); has_sums = false; continue; }
            }
            n += 1;
            nfull++;
            T X, Y;
            BSRef<T>::orbit(R, w, X, Y);
            T Xa = cst<T>(0.f), Xb = cst<T>(0.f), Ya = cst<T>(0.f), Yb = cst<T>(0.f);
            if (hess && !dyn) BSRef<T>::hess(R, w, Xa, Xb, Ya, Yb);
            bool taken = false;
            if constexpr (IsDouble<T>::value && FL == 1) {
                if (below) {
                    if (dyn && (dbits(X) | dbits(Y)) == 0) taken = bs_ship_crit(hess, xn, yn, h, a, b);
                    else if (AXIS) taken = bs_ship_deep(hess, xn, yn, h, X, Y, Xa, Xb, Ya, Yb, a, b);
                }
                if (!taken) {
                    double xs = XX_last, ys = YY_last;
                    if (!has_sums) {
                        xs = (d_is0(X) & !d_is0(xn)) ? xn : d_add_here(X, xn);
                        ys = (d_is0(Y) & !d_is0(yn)) ? yn : d_add_here(Y, yn);
                    }
                    taken = bs_step_ship<AXIS>(hess, xn, yn, h, X, Y, xs, ys, Xa, Xb, Ya, Yb, a, b);
                }
            }
            if (!taken) {
                if (hess) bs_hess<T>(flavor, h, xn, yn, X, Y, Xa, Xb, Ya, Yb);
                bs_zn<T>(flavor, xn, yn, X, Y, a, b);
            }
            if (n >= C.max_iter) { stop = 0; break; }
            w += 1;
            if (w >= order) w = 0;
        }
        if constexpr (XR_FORM) {
            // the Xrange branch's tests (perturbation.py:1627-1731): escape on
            // the standard values; rebase when the reference diverges from
            // the standard sum; the dynamic rebase tested componentwise on the
            // standard values, then confirmed with |Z + z|^2 <= |z|^2 in
            // Xrange (with the side table's value of the orbit where it holds
            // one) -- a refused confirmation leaves bool_dyn_rebase set
            const double2 Zs = __ldg(&R.Zn[w]);
            const double xs = to_d(xn), ys = to_d(yn);
            const double XXd = xs + Zs.x, YYd = ys + Zs.y;
            if (bs > 0) S.take(n, bs, cx(XXd, YYd));
            if (fsg_escaped(C, cx(XXd, YYd))) { stop = 1; break; }
            if (w >= div_iter - 1) {
                xn = from_d<T>(XXd); yn = from_d<T>(YYd);
                if (hess) {
                    T Ha, Hb, Hc, Hd;
                    BSRef<T>::hess(R, w, Ha, Hb, Hc, Hd);
                    h[0] += Ha; h[1] += Hb; h[2] += Hc; h[3] += Hd;
                }
                w = 0; nreb++; continue;
            }
            dyn = d_abs_le(XXd, xs) && d_abs_le(YYd, ys);
            if (dyn) {
                T Xt, Yt;
                const bool tab = BSRef<T>::table(R, w, Xt, Yt);
                const T XXx = tab ? xn + Xt : xf_add_s(xn, Zs.x);
                const T YYx = tab ? yn + Yt : xf_add_s(yn, Zs.y);
                if (xf_le(XXx * XXx + YYx * YYx, xn * xn + yn * yn)) {
                    xn = XXx; yn = YYx;
                    if (hess) {
                        T Ha, Hb, Hc, Hd;
                        BSRef<T>::hess(R, w, Ha, Hb, Hc, Hd);
                        h[0] += Ha; h[1] += Hb; h[2] += Hc; h[3] += Hd;
                    }
                    w = 0; nreb++; continue;
                }
            }
            continue;
        }
        T Xs, Ys;
        BSRef<T>::orbit(R, w, Xs, Ys);
        T XX, YY;
        if constexpr (IsDouble<T>::value) {
            XX = d_add_far(xn, Xs);
            YY = d_add_far(yn, Ys);
            XX_last = XX; YY_last = YY;
            has_sums = true;
        } else {
            XX = xn + Xs; YY = yn + Ys;
        }
        if constexpr (ORB_FORM) {
            const double XXd = to_d(XX), YYd = to_d(YY);
            if (bs > 0) S.take(n, bs, cx(XXd, YYd));             // :1641-1651
            if (fsg_escaped(C, cx(XXd, YYd))) { stop = 1; break; }
        } else {
            if (fr_escaped(XX, YY, M2f, C.M2)) { stop = 1; break; }
        }
        if (w >= div_iter - 1) {
            xn = XX; yn = YY;
            has_sums = false;
            if (hess) {
                T Ha, Hb, Hc, Hd;
                BSRef<T>::hess(R, w, Ha, Hb, Hc, Hd);
                h[0] = bs_add<T, FL>(h[0], Ha); h[1] = bs_add<T, FL>(h[1], Hb);
                h[2] = bs_add<T, FL>(h[2], Hc); h[3] = bs_add<T, FL>(h[3], Hd);
            }
            w = 0; nreb++; continue;
        }
        dyn = abs_le(XX, xn) && abs_le(YY, yn);
        if (dyn) {
            xn = XX; yn = YY;
            has_sums = false;
            if (hess) {
                T Ha, Hb, Hc, Hd;
                BSRef<T>::hess(R, w, Ha, Hb, Hc, Hd);
                h[0] = bs_add<T, FL>(h[0], Ha); h[1] = bs_add<T, FL>(h[1], Hb);
                h[2] = bs_add<T, FL>(h[2], Hc); h[3] = bs_add<T, FL>(h[3], Hd);
            }
            w = 0; nreb++; continue;
        }
        if constexpr (FR_FORM) {
            // the frame form takes over while the deltas stay below 2^11 and
            // the next step can run there
            if (max(xn.e, yn.e) <= 10 && (__ldg(&R.bs_at[3 * (size_t)w]).x & 5)) {
                frame_in(Fm, xn, yn, h);
                frm = true;
            }
        }
    }
    // end of iterations (:1745-1757): the Xrange branch adds the standard
    // orbit value to the Xrange delta
    double xo, yo;
    if constexpr (XR_FORM) {
        const double2 Zs = __ldg(&R.Zn[w]);
        xo = to_d(xf_add_s(xn, Zs.x)); yo = to_d(xf_add_s(yn, Zs.y));
    } else {
        T Xe, Ye;
        BSRef<T>::orbit(R, w, Xe, Ye);
        xo = to_d(xn + Xe); yo = to_d(yn + Ye);
    }
    double hd[4] = {0., 0., 0., 0.};
    if (hess) {
        // the Hessian in the tile's unit: the reference's scale times 2^dzs
        T Ha, Hb, Hc, Hd;
        BSRef<T>::hess(R, w, Ha, Hb, Hc, Hd);
        hd[0] = to_d(scale2(h[0] + Ha, Tl.dzs)); hd[1] = to_d(scale2(h[1] + Hb, Tl.dzs));
        hd[2] = to_d(scale2(h[2] + Hc, Tl.dzs)); hd[3] = to_d(scale2(h[3] + Hd, Tl.dzs));
        if (Tl.proj) {
            // Expmap (perturbation.py:1772-1776)
            const double m = fsg_dzndc_modifier(Tl, ip);
            hd[0] *= m; hd[1] *= m; hd[2] *= m; hd[3] *= m;
        }
    }
    double *Z = (double *)Tl.Z;
    if (bs > 0) {
        // :1778-1787: the reference replays with AA = a + Re(Z_1) and
        // BB = b + Im(Z_1) = b - b_ref (kept as is)
        const double2 Z1 = __ldg(&R.Zn[1]);
        const double AA = to_d(a) + Z1.x, BB = to_d(b) + Z1.y;
        double xr = S.z2.x, yr = S.z2.y;
        for (int i2 = S.i2; i2 < n - bs; i2++) {
            double nx_, ny_;
            bs_map(flavor, xr, yr, AA, BB, nx_, ny_);
            xr = nx_; yr = ny_;
        }
        Z[(long long)Tl.i_orb * np + ip] = xr;
        Z[(long long)(Tl.i_orb + 1) * np + ip] = yr;
    }
    Z[ip] = xo; Z[np + ip] = yo;
    if (hess) { Z[2 * np + ip] = hd[0]; Z[3 * np + ip] = hd[1]; Z[4 * np + ip] = hd[2]; Z[5 * np + ip] = hd[3]; }
    if (Tl.U) Tl.U[ip] = w;
    Tl.stop_iter[ip] = n; Tl.stop_reason[ip] = stop;
    double absd = 0.5 * (hypot(hd[0] + hd[3], hd[1] - hd[2]) + hypot(hd[0] - hd[3], hd[1] + hd[2]));
    fsg_epilogue(Tl, C, ip, cx(xo, yo), absd, n);
    return n;
}

// DENSE: the FP32 + exponent kernels hold three 256-thread blocks per SM (at most 85
// registers a thread), or four (64, with spills) for images that three do not hold
// at once: short chains of FP32 and integer operations want warps more than
// registers -- flavor 1, 640^2 pixels of a period-12 nucleus to 20000 iterations,
// takes 45.5 ms with four, 48.0 with three, 48.9 with five, 60.6 with two; images of
// 150^2 and 300^2 take 1 to 5 % longer with four, of 450^2 and 600^2 5 to 14 % less,
// but for flavor 5, whose views spend more in the fr steps, which spill (31 to 34
// ms with three, 35 with four).  The other kernels hold two (128): flavor 1 in the
// double form, 255^2 pixels of the period-12 nucleus to 20000 iterations, took 68 ms
// with them before bs_ship_deep (36 with it), 95 ms at its own 156 registers and one
// block, 73 ms at 80 with spills
template <class T, int FL, bool AXIS, bool DENSE>
__global__ void __launch_bounds__(256, DENSE ? 4 : IsFr<T>::value ? 3 : 2)
k_perturb_bs(WorkDev W, CalcDev C) {
    // sized at launch: per-thread statistics (64-bit sums would hold 8 registers
    // in the loop), then the pixel offsets of the launch's tiles
    extern __shared__ unsigned long long bs_smem[];
    unsigned long long *acc = bs_smem + threadIdx.x;           // acc[k * blockDim.x]
    long long *s_start = (long long *)(bs_smem + 4 * blockDim.x);
    const int nb = blockDim.x;
    for (int k = 0; k < 4; k++) acc[k * nb] = 0ULL;
    fsg_load_starts(W, s_start);
    int t; long long ip;
    while (true) {
        if (!fsg_claim_poll(W, s_start, t, ip)) break;
        unsigned nfull = 0, nbla = 0, nreb = 0;
        const int n = pixel_bs<T, FL, AXIS>(W.tiles[t], C, ip, nfull, nbla, nreb);
        fsg_account(W, (unsigned long long)n);
        acc[0] += (unsigned long long)n;
        acc[nb] += nfull;
        acc[2 * nb] += nbla;
        acc[3 * nb] += nreb;
    }
    fsg_flush_stats(W, acc[0], acc[nb], acc[2 * nb], acc[3 * nb]);
}
