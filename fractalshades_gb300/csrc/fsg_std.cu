// fsg_std.cu -- standard (non-perturbation) escape-time loops, FP64.
//
// Power-2 Mandelbrot: core.py:2935-3004 numba_cycles / numba_iterate and
// models/mandelbrot_M2.py:309-334 iterate_once; power-n Mandelbrot:
// models/mandelbrot_Mn.py:317-355.  Burning Ship family:
// core.py:3007-3056 numba_iterate_BS and models/burning_ship.py:350-434.
// The reference compiles these without fastmath, so this file is built with
// -fmad=false: each operation rounds once, in the order of the reference.
#include "fsg_internal.cuh"

__device__ __forceinline__ double sgn(double x) { return x < 0. ? -1. : 1.; }

// core.py:3161-3194 c_from_pix, Cartesian projection
__device__ __forceinline__ double2 std_c(const TileDev &T, long long ip) {
    double2 pp = fsg_pixel(T, ip);
    double px = pp.x, py = pp.y;
    double x1 = T.lin[0] * px + T.lin[1] * py;
    double y1 = T.lin[2] * px + T.lin[3] * py;
    return cadd(cx(T.cre, T.cim), rmul(T.dx, cx(x1, y1)));
}

#define FSG_STD_CHUNK 16        // steps between two block-level compaction checks
#define FSG_STD_REFILL 4        // steps between two refills of a warp's idle lanes
#define FSG_STD_CANCEL 64       // chunks between two reads of the cancel flag

// The models.  A pixel's state is its Px: what a lane iterates, what waits in
// a warp's queue and what the block compaction moves.
//   start: c known, the state of z_0 = 0 in place (n = 0); takes the first
//          steps of an ordinary pixel (all lanes of a warp run it together);
//   step:  one iteration; products by fsg_soft.cuh, and by the multiplies
//          (step_full, the reference's operations one by one, out of line)
//          where a factor is out of their range (in_range) or a product is left
//          open;
//   stop:  the tests after it: the stop reason, -1 to go on;
//   store: the outputs.
// OPT: the optional outputs d2zndc2 (mandelbrot_M2.py:316-317) and the orbit
// point n - backshift (core.py:2965-3004).
template <bool OPT> struct StdOpt { double2 d2; OrbitSnap<double2> S; };
template <> struct StdOpt<false> {};

template <bool OPT>
__device__ __forceinline__ void std_opt_init(StdOpt<OPT> &o, const CalcDev &C) {
    if constexpr (OPT) { o.d2 = cx(0., 0.); o.S.init(C.backshift, cx(0., 0.)); }
}
template <bool OPT>
__device__ __forceinline__ void std_opt_take(StdOpt<OPT> &o, const CalcDev &C, int n, double2 z) {
    if constexpr (OPT) { if (C.backshift > 0) o.S.take(n, C.backshift, z); }
}

template <class Mdl>
static __device__ __noinline__ typename Mdl::Px std_step_full(typename Mdl::Px p, const CalcDev &C) {
    Mdl::step_full(p, C);
    return p;
}

struct CoopLane { unsigned k, neg; bool add; double g; };

// Power-2 and power-n Mandelbrot: the complex state
template <bool OPT>
struct StdPx { double2 c, zn, dzndz, dzndc; StdOpt<OPT> o; long long ip; int t, n; };

template <bool OPT>
struct StdMandel {
    typedef StdPx<OPT> Px;
    static __device__ __forceinline__ void init(Px &p, const CalcDev &C, double2 c) {
        p.c = c; p.zn = cx(0., 0.); p.dzndz = p.zn; p.dzndc = p.zn; p.n = 0;
        std_opt_init<OPT>(p.o, C);
    }
    static __device__ __forceinline__ bool in_range(const Px &p, const CalcDev &C) {
        bool ok = dfac_ok(p.zn) & dfac_ok(p.dzndz) & dfac_ok(p.dzndc);
        if constexpr (OPT) { if (C.d2) ok &= dfac_ok(p.o.d2); }
        return ok;
    }
    static __device__ __forceinline__ int stop(const Px &p, const CalcDev &C) {
        if (fsg_escaped(C, p.zn)) return 1;
        if (fsg_stationary(C, p.dzndz)) return 2;
        return -1;
    }
    static __device__ __forceinline__ void store_z(const Px &p, const TileDev &T) {
        const long long np = (long long)T.nx * T.ny;
        double2 *Z = (double2 *)T.Z;
        Z[p.ip] = p.zn; Z[np + p.ip] = p.dzndz; Z[2 * np + p.ip] = p.dzndc;
    }
};

// models/mandelbrot_M2.py:309-334 iterate_once
template <bool OPT>
struct StdM2 : StdMandel<OPT> {
    typedef StdPx<OPT> Px;
    static __device__ __forceinline__ void step_full(Px &p, const CalcDev &C) {
        if constexpr (OPT) {
            if (C.d2) p.o.d2 = rmul2(cadd(cmul(p.o.d2, p.zn), csq(p.dzndc)));
        }
        p.dzndc = caddr(cmul(rmul2(p.dzndc), p.zn), 1.);
        p.dzndz = cmul(rmul2(p.dzndz), p.zn);
        p.zn = cadd(csq(p.zn), p.c);
    }
    static __device__ __forceinline__ void step(Px &p, const CalcDev &C) {
        bool ok = dfac_ok(p.zn) & dfac_ok(p.dzndz) & dfac_ok(p.dzndc);
        const cfac z = cfac_of(p.zn), c2 = cfac_of(p.dzndc, 1);
        double2 d2 = cx(0., 0.);
        if constexpr (OPT) {
            if (C.d2) {
                ok &= dfac_ok(p.o.d2);
                d2 = rmul2(cadd(cfac_mul(cfac_of(p.o.d2), z, ok), cfac_sq(cfac_of(p.dzndc), ok)));
            }
        }
        const double2 sq = cfac_sq(z, ok);
        const double2 dz = cfac_mul(cfac_of(p.dzndz, 1), z, ok);
        double2 dc = cfac_mul(c2, z, ok);
        dc.x += 1.;
        if (ok) {
            p.zn = cadd(sq, p.c); p.dzndz = dz; p.dzndc = dc;
            if constexpr (OPT) { if (C.d2) p.o.d2 = d2; }
        } else {
            p = std_step_full<StdM2<OPT>>(p, C);
        }
    }
    // z_1 = c and dz_1 = dc_1 = 1, z_2 = c^2 + c, dz_2 = 2 c and dc_2 = 2 c + 1
    // for c in the range of the integer products (elsewhere the pixel starts at
    // n = 0); with d2zndc2 up to three plain steps, those before the last one
    static __device__ __forceinline__ void start(Px &p, const CalcDev &C) {
        Px s = p;
        if (OPT && C.d2) {
            for (int n = 1; n <= min(3, C.max_iter - 1); n++) {
                step_full(s, C);
                if (n == 1) s.dzndz = cx(1., 0.);
                std_opt_take<OPT>(s.o, C, n, s.zn);
                if (StdMandel<OPT>::stop(s, C) >= 0) break;
                s.n = n;
                p = s;
            }
            return;
        }
        bool ok = dfac_ok(p.c) && C.max_iter > 2;
        s.zn = p.c; s.dzndz = cx(1., 0.);
        ok &= StdMandel<OPT>::stop(s, C) < 0;
        std_opt_take<OPT>(s.o, C, 1, s.zn);
        s.zn = cadd(cfac_sq(cfac_of(p.c), ok), p.c);
        s.dzndz = cx(d_twice(p.c.x), d_twice(p.c.y));
        s.dzndc = cx(s.dzndz.x + 1., s.dzndz.y);
        ok &= StdMandel<OPT>::stop(s, C) < 0;
        std_opt_take<OPT>(s.o, C, 2, s.zn);
        s.n = 2;
        if (ok) p = s;
    }
    // A step by eight lanes of one pixel (std_coop): lane `role` holds one
    // component `own` -- 0, 1 z; 2, 3 dz/dz; 4, 5 dz/dc -- and sees z = (x, y)
    // and its partner `pr`, the other part of its pair.  Every component is
    // own x -+ pr y (doubled for the derivatives), and what is added to it.
    static constexpr bool kCoop = !OPT;
    static constexpr bool kPlain = OPT;                  // std_plain_chunk
    static __device__ __forceinline__ double coop_get(const Px &p, int role) {
        return role == 0 ? p.zn.x : role == 1 ? p.zn.y : role == 2 ? p.dzndz.x
               : role == 3 ? p.dzndz.y : role == 4 ? p.dzndc.x : p.dzndc.y;
    }
    static __device__ __forceinline__ int coop_partner(int role) { return role ^ 1; }
    // what the fast form needs of a lane: k the doubling, neg the sign of the
    // second product, g what is added (add)
    static __device__ __forceinline__ CoopLane coop_lane(const Px &p, const CalcDev &, int role) {
        CoopLane L;
        L.k = role < 2 ? 0u : 0x00100000u;
        L.neg = (role & 1) ? 0u : 0x80000000u;
        L.add = (role & 6) != 2;
        L.g = role == 0 ? p.c.x : role == 1 ? p.c.y : role == 4 ? 1. : 0.;
        return L;
    }
    static __device__ __forceinline__ double coop_fast(double own, double pr, double x, double y,
                                                       const CoopLane &L, const CalcDev &, int, int,
                                                       bool &ok) {
        dfac fx = dfac_of(x), fy = dfac_of(y);
        fx.s += L.k; fy.s += L.k ^ L.neg;
        const double u = dfac_mul0(dfac_of0(own), fx, ok) + dfac_mul0(dfac_of0(pr), fy, ok);
        const double w = u + L.g;
        return L.add ? w : u;
    }
    // step_full for one lane
    static __device__ __forceinline__ double coop_full(double own, double pr, double x, double y,
                                                       const Px &p, const CoopLane &, const CalcDev &,
                                                       int role, int n) {
        const bool im = role & 1;
        double2 a = im ? cx(pr, own) : cx(own, pr);
        if (role >= 2) a = rmul2(a);
        const double2 m = cmul(a, cx(x, y));
        const double u = im ? m.y : m.x;
        if (role == 0) return u + p.c.x;
        if (role == 1) return u + p.c.y;
        if (role >= 4) return u + (role == 4 ? 1. : 0.);
        return n == 1 ? (role == 2 ? 1. : 0.) : u;
    }
    // whether the tests after a step need more than exponents
    static __device__ __forceinline__ bool coop_near(double own, double pr, double x, double y,
                                                     const CalcDev &C, int role) {
        return (d_mag_hi(cx(x, y)) >= C.esc.lo) | ((role == 2) & (d_mag_hi(cx(own, pr)) < C.stat.hi));
    }
    // the stop reason, the same in the pixel's eight lanes
    static __device__ __forceinline__ int coop_stop(double own, double pr, double x, double y,
                                                    const CalcDev &C, int base, int role) {
        const bool still = role == 2 && fsg_stationary(C, cx(own, pr));
        const unsigned b = __ballot_sync(0xffffffffu, still);
        if (fsg_escaped(C, cx(x, y))) return 1;
        return (b >> (base + 2) & 1u) ? 2 : -1;
    }
    static __device__ __forceinline__ void coop_store(double own, const Px &p, const TileDev &T, int role) {
        const long long np = (long long)T.nx * T.ny;
        ((double *)T.Z)[2 * ((role >> 1) * np + p.ip) + (role & 1)] = own;
    }
    static __device__ __forceinline__ void store(const Px &p, const TileDev &T, const CalcDev &C) {
        StdMandel<OPT>::store_z(p, T);
        if constexpr (OPT) {
            const long long np = (long long)T.nx * T.ny;
            double2 *Z = (double2 *)T.Z;
            if (C.d2) Z[3 * np + p.ip] = p.o.d2;
            if (C.backshift > 0) {
                double2 zo = p.o.S.z2;
                for (int i2 = p.o.S.i2; i2 < p.n - C.backshift; i2++) zo = cadd(csq(zo), p.c);   // M2_iterate
                Z[(long long)T.i_orb * np + p.ip] = zo;
            }
        }
    }
};

// z^k by the integer products, in mn_ipow's order (its first product, by
// 1 + 0 i, is its factor itself: the factors are finite and not 0)
__device__ __forceinline__ double2 ipow_soft(double2 a, int n, bool &ok) {
    if (n == 1) return a;
    const cfac fa = cfac_of(a);
    if (n == 2) return cfac_sq(fa, ok);
    if (n == 3) {
        const double2 q = cfac_sq(fa, ok);
        ok &= dfac_ok(q);
        return cfac_mul(fa, cfac_of(q), ok);
    }
    double2 acc = cx(1., 0.), p = a;
    bool one = true;
    int mask = 1;
    for (;;) {
        ok &= dfac_ok(p);
        if (n & mask) {
            if (one) { acc = p; one = false; }
            else { ok &= dfac_ok(acc); acc = cfac_mul(cfac_of(acc), cfac_of(p), ok); }
        }
        mask <<= 1;
        if (n < mask) break;
        p = cfac_sq(cfac_of(p), ok);
    }
    return acc;
}

// models/mandelbrot_Mn.py:317-355 iterate_once: z^(n-1) once per step,
// z^n = z^(n-1) z
template <bool OPT>
struct StdMn : StdMandel<OPT> {
    typedef StdPx<OPT> Px;
    static constexpr bool kCoop = false;
    static constexpr bool kPlain = true;
    static __device__ __forceinline__ void step_full(Px &p, const CalcDev &C) {
        const int nexp = C.nexp;
        const double deg = (double)nexp;
        double2 zm1, zm;
        bool d2_on = false;
        if constexpr (OPT) {
            if (C.d2) {
                d2_on = true;
                // mandelbrot_Mn.py:325-333; the reference's recurrence
                // multiplies by dzndz where d/dc of n z^(n-1) dzndc has dzndc
                double2 zm2 = mn_ipow(p.zn, nexp - 2);
                zm1 = cmul(zm2, p.zn);
                zm = cmul(zm1, p.zn);
                p.o.d2 = rmul(deg, cadd(cmul(p.o.d2, zm1),
                                        cmul(cmul(rmul((double)(nexp - 1), p.dzndz), p.dzndc), zm2)));
            }
        }
        if (!d2_on) {
            zm1 = mn_ipow(p.zn, nexp - 1);
            zm = cmul(zm1, p.zn);
        }
        p.dzndc = caddr(cmul(rmul(deg, p.dzndc), zm1), 1.);
        p.dzndz = cmul(rmul(deg, p.dzndz), zm1);
        p.zn = cadd(zm, p.c);
    }
    // deg * z by the integer products (by a small integer: ties are common)
    static __device__ __forceinline__ double2 scaled(const dfac &deg, double2 z) {
        return cx(dfac_mul_ties(deg, dfac_of(z.x)), dfac_mul_ties(deg, dfac_of(z.y)));
    }
    static __device__ __forceinline__ void step(Px &p, const CalcDev &C) {
        const int nexp = C.nexp;
        bool ok = dfac_ok(p.zn) & dfac_ok(p.dzndz) & dfac_ok(p.dzndc);
        const dfac deg = dfac_of((double)nexp);
        double2 zm1, d2 = cx(0., 0.);
        bool d2_on = false;
        if constexpr (OPT) {
            if (C.d2 && nexp > 2) {
                d2_on = true;
                const double2 zm2 = ipow_soft(p.zn, nexp - 2, ok);
                ok &= dfac_ok(zm2) & dfac_ok(p.o.d2);
                zm1 = cfac_mul(cfac_of(zm2), cfac_of(p.zn), ok);
                ok &= dfac_ok(zm1);
                const double2 u = scaled(dfac_of((double)(nexp - 1)), p.dzndz);
                ok &= dfac_ok(u);
                const double2 v = cfac_mul(cfac_of(u), cfac_of(p.dzndc), ok);
                ok &= dfac_ok(v);
                const double2 w = cadd(cfac_mul(cfac_of(p.o.d2), cfac_of(zm1), ok),
                                       cfac_mul(cfac_of(v), cfac_of(zm2), ok));
                ok &= dfac_ok(w);
                d2 = scaled(deg, w);
            } else if (C.d2) {
                // n = 2: z^0 = 1 leaves its factors as they are
                ok &= dfac_ok(p.o.d2);
                const double2 w = cadd(cfac_mul(cfac_of(p.o.d2), cfac_of(p.zn), ok),
                                       cfac_mul(cfac_of(p.dzndz), cfac_of(p.dzndc), ok));
                ok &= dfac_ok(w);
                d2 = scaled(deg, w);
            }
        }
        if (!d2_on) zm1 = ipow_soft(p.zn, nexp - 1, ok);
        ok &= dfac_ok(zm1);
        const cfac fm = cfac_of(zm1);
        const double2 zm = cfac_mul(fm, cfac_of(p.zn), ok);
        const double2 ec = scaled(deg, p.dzndc), ez = scaled(deg, p.dzndz);
        ok &= dfac_ok(ec) & dfac_ok(ez);
        double2 dc = cfac_mul(cfac_of(ec), fm, ok);
        dc.x += 1.;
        const double2 dz = cfac_mul(cfac_of(ez), fm, ok);
        if (ok) {
            p.zn = cadd(zm, p.c); p.dzndz = dz; p.dzndc = dc;
            if constexpr (OPT) { if (C.d2) p.o.d2 = d2; }
        } else {
            p = std_step_full<StdMn<OPT>>(p, C);
        }
    }
    // z_1 = c, dz_1 = dc_1 = 1; dz_2 = n c^(n-1), dc_2 = dz_2 + 1,
    // z_2 = c^n + c; with d2zndc2 up to three plain steps
    static __device__ __forceinline__ void start(Px &p, const CalcDev &C) {
        Px s = p;
        if (OPT && C.d2) {
            for (int n = 1; n <= min(3, C.max_iter - 1); n++) {
                step_full(s, C);
                if (n == 1) s.dzndz = cx(1., 0.);
                std_opt_take<OPT>(s.o, C, n, s.zn);
                if (StdMandel<OPT>::stop(s, C) >= 0) break;
                s.n = n;
                p = s;
            }
            return;
        }
        bool ok = dfac_ok(p.c) && C.max_iter > 2;
        s.zn = p.c; s.dzndz = cx(1., 0.);
        ok &= StdMandel<OPT>::stop(s, C) < 0;
        std_opt_take<OPT>(s.o, C, 1, s.zn);
        const double2 zm1 = ipow_soft(p.c, C.nexp - 1, ok);
        ok &= dfac_ok(zm1);
        s.zn = cadd(cfac_mul(cfac_of(zm1), cfac_of(p.c), ok), p.c);
        s.dzndz = scaled(dfac_of((double)C.nexp), zm1);
        s.dzndc = cx(s.dzndz.x + 1., s.dzndz.y);
        ok &= StdMandel<OPT>::stop(s, C) < 0;
        std_opt_take<OPT>(s.o, C, 2, s.zn);
        s.n = 2;
        if (ok) p = s;
    }
    static __device__ __forceinline__ void store(const Px &p, const TileDev &T, const CalcDev &C) {
        StdMandel<OPT>::store_z(p, T);
        if constexpr (OPT) {
            const long long np = (long long)T.nx * T.ny;
            double2 *Z = (double2 *)T.Z;
            if (C.d2) Z[3 * np + p.ip] = p.o.d2;
            if (C.backshift > 0) {
                double2 zo = p.o.S.z2;
                for (int i2 = p.o.S.i2; i2 < p.n - C.backshift; i2++)
                    zo = cadd(mn_ipow(zo, C.nexp), p.c);   // Mn_iterate
                Z[(long long)T.i_orb * np + p.ip] = zo;
            }
        }
    }
};

// Burning Ship family: models/burning_ship.py:350-434, core.py:3007-3056
template <bool OPT>
struct StdBSPx { double a, b, X, Y, Xa, Xb, Ya, Yb; StdOpt<OPT> o; long long ip; int t, n; };

template <bool OPT>
struct StdBS {
    typedef StdBSPx<OPT> Px;
    static __device__ __forceinline__ void init(Px &p, const CalcDev &C, double2 c) {
        p.a = c.x; p.b = c.y;
        p.X = 0.; p.Y = 0.; p.Xa = 0.; p.Xb = 0.; p.Ya = 0.; p.Yb = 0.; p.n = 0;
        std_opt_init<OPT>(p.o, C);
    }
    static __device__ __forceinline__ int stop(const Px &p, const CalcDev &C) {
        return fsg_escaped(C, cx(p.X, p.Y)) ? 1 : -1;
    }
    static __device__ __forceinline__ void step_full(Px &p, const CalcDev &C) {
        const int flavor = C.flavor;
        const double X = p.X, Y = p.Y, a = p.a, b = p.b;
        const double dXdA = p.Xa, dXdB = p.Xb, dYdA = p.Ya, dYdB = p.Yb;
        double nX, nY, nXa, nXb, nYa, nYb;
        if (flavor == 1) {
            nX = X * X - Y * Y + a;
            nY = 2. * fabs(X * Y) - b;
            nXa = 2. * (X * dXdA - Y * dYdA) + 1.;
            nXb = 2. * (X * dXdB - Y * dYdB);
            nYa = 2. * (fabs(X) * sgn(Y) * dYdA + sgn(X) * dXdA * fabs(Y));
            nYb = 2. * (fabs(X) * sgn(Y) * dYdB + sgn(X) * dXdB * fabs(Y)) - 1.;
        } else if (flavor == 2) {
            nX = X * X - Y * Y + a;
            nY = 2. * X * fabs(Y) - b;
            nXa = 2. * (X * dXdA - Y * dYdA) + 1.;
            nXb = 2. * (X * dXdB - Y * dYdB);
            nYa = 2. * (X * sgn(Y) * dYdA + dXdA * fabs(Y));
            nYb = 2. * (X * sgn(Y) * dYdB + dXdB * fabs(Y)) - 1.;
        } else if (flavor == 3) {
            nX = X * X - Y * fabs(Y) + a;
            nY = 2. * X * Y - b;
            nXa = 2. * (X * dXdA - fabs(Y) * dYdA) + 1.;
            nXb = 2. * (X * dXdB - fabs(Y) * dYdB);
            nYa = 2. * (dXdA * Y + X * dYdA);
            nYb = 2. * (dXdB * Y + X * dYdB) - 1.;
        } else if (flavor == 4) {
            double q = X * X - Y * Y;
            nX = fabs(q) + a;
            nY = 2. * X * Y - b;
            nXa = 2. * sgn(q) * (X * dXdA - Y * dYdA);
            nXb = 2. * sgn(q) * (X * dXdB - Y * dYdB);
            nYa = 2. * (dXdA * Y + X * dYdA);
            nYb = 2. * (dXdB * Y + X * dYdB) - 1.;
        } else {
            double q = X * X - Y * Y;
            nX = fabs(q) + a;
            nY = 2. * fabs(X * Y) - b;
            nXa = 2. * sgn(q) * (X * dXdA - Y * dYdA);
            nXb = 2. * sgn(q) * (X * dXdB - Y * dYdB);
            nYa = 2. * (fabs(X) * sgn(Y) * dYdA + sgn(X) * dXdA * fabs(Y));
            nYb = 2. * (fabs(X) * sgn(Y) * dYdB + sgn(X) * dXdB * fabs(Y)) - 1.;
        }
        p.X = nX; p.Y = nY; p.Xa = nXa; p.Xb = nXb; p.Ya = nYa; p.Yb = nYb;
    }
    // With X and Y in the range of the integer products and every derivative
    // there or 0 (flavors 4 and 5 keep dX/da = dY/da = 0): the products by
    // +-1 change signs, those by 2 exponents, and each remaining product and
    // sum rounds as in step_full.
    static __device__ __forceinline__ bool in_range(const Px &p, const CalcDev &) {
        return dfac_ok(p.X) & dfac_ok(p.Y) & dfac_ok0(p.Xa) & dfac_ok0(p.Xb) & dfac_ok0(p.Ya)
               & dfac_ok0(p.Yb);
    }
    static __device__ __forceinline__ void step(Px &p, const CalcDev &C) {
        const int flavor = C.flavor;
        bool ok = dfac_ok(p.X) & dfac_ok(p.Y) & dfac_ok0(p.Xa) & dfac_ok0(p.Xb)
                  & dfac_ok0(p.Ya) & dfac_ok0(p.Yb);
        // 2 X and 2 Y, the factors of every derivative
        const dfac X = dfac_of(p.X), Y = dfac_of(p.Y), X2 = dfac_of(p.X, 1), Y2 = dfac_of(p.Y, 1);
        const dfac Xa = dfac_of0(p.Xa), Xb = dfac_of0(p.Xb), Ya = dfac_of0(p.Ya), Yb = dfac_of0(p.Yb);
        const unsigned sX = X.s & 0x80000000u, sY = Y.s & 0x80000000u;
        const bool ship = flavor == 1 || flavor == 5, fold = flavor >= 4;
        const double xx = dfac_mul(X, X, ok), xy2 = dfac_mul(X2, Y, ok), yy = dfac_mul(Y, Y, ok);
        // X^2 - Y^2 (flavor 3: X^2 - Y |Y|)
        const double q = xx - (flavor == 3 ? d_flip(yy, sY) : yy);
        const unsigned sq = d_lt0(q) ? 0x80000000u : 0u;
        const double nX = (fold ? d_abs(q) : q) + p.a;
        // |X Y| 2, X |Y| 2 or X Y 2
        const double nY = d_flip(xy2, ship ? sX ^ sY : flavor == 2 ? sY : 0u) - p.b;
        dfac Yf = Y2;
        if (flavor == 3) Yf.s ^= sY;                     // |Y|
        double xa = dfac_mul0(X2, Xa, ok) - dfac_mul0(Yf, Ya, ok);
        double xb = dfac_mul0(X2, Xb, ok) - dfac_mul0(Yf, Yb, ok);
        if (fold) { xa = d_flip(xa, sq); xb = d_flip(xb, sq); }
        else xa += 1.;
        // the factor of dY: |X| sgn(Y), X sgn(Y) or X; of dX: sgn(X) |Y|, |Y| or Y
        dfac P = X2, R = Y2;
        if (ship) { P.s ^= sX ^ sY; R.s ^= sX ^ sY; }
        else if (flavor == 2) { P.s ^= sY; R.s ^= sY; }
        const double ya = dfac_mul0(P, Ya, ok) + dfac_mul0(R, Xa, ok);
        const double yb = dfac_mul0(P, Yb, ok) + dfac_mul0(R, Xb, ok) - 1.;
        if (ok) {
            p.X = nX; p.Y = nY; p.Xa = xa; p.Xb = xb; p.Ya = ya; p.Yb = yb;
        } else {
            p = std_step_full<StdBS<OPT>>(p, C);
        }
    }
    static __device__ __forceinline__ void start(Px &p, const CalcDev &C) {
        // n = 1: X = a, Y = -b from zeros, in the plain form (one step's
        // operations for 32 pixels)
        Px s = std_step_full<StdBS<OPT>>(p, C);
        std_opt_take<OPT>(s.o, C, 1, cx(s.X, s.Y));
        s.n = 1;
        if (C.max_iter > 1 && stop(s, C) < 0) p = s;
    }
    // Eight lanes of one pixel (std_coop): 0 X, 1 Y, 2 dX/da, 3 dX/db, 4 dY/da,
    // 5 dY/db; the partners are X and Y and the derivatives by one coordinate.
    // Every component is own X' +- pr Y' with X' = +-X or +-2 X, Y' likewise.
    static constexpr bool kCoop = !OPT;
    static constexpr bool kPlain = true;
    static __device__ __forceinline__ double coop_get(const Px &p, int role) {
        return role == 0 ? p.X : role == 1 ? p.Y : role == 2 ? p.Xa : role == 3 ? p.Xb
               : role == 4 ? p.Ya : p.Yb;
    }
    static __device__ __forceinline__ int coop_partner(int role) {
        return role < 2 ? 1 - role : role < 4 ? role + 2 : role - 2;
    }
    static __device__ __forceinline__ CoopLane coop_lane(const Px &p, const CalcDev &C, int role) {
        CoopLane L;
        L.k = role == 0 ? 0u : 0x00100000u;
        L.neg = role < 4 ? 0x80000000u : 0u;
        L.g = role == 0 ? p.a : role == 1 ? -p.b : role == 2 ? 1. : -1.;
        L.add = role < 2 || (role == 2 && C.flavor < 4) || role == 5;
        return L;
    }
    static __device__ __forceinline__ double coop_fast(double own, double pr, double x, double y,
                                                       const CoopLane &L, const CalcDev &C, int base,
                                                       int role, bool &ok) {
        const int flavor = C.flavor;
        const bool ship = flavor == 1 || flavor == 5, fold = flavor >= 4;
        const unsigned sx = d_hi(x) & 0x80000000u, sy = d_hi(y) & 0x80000000u;
        // signs of the factors: dY's are |X| sgn(Y), X sgn(Y) or X (with sgn(X)
        // |Y|, |Y| or Y); flavor 3 has |Y| in dX and in X
        const unsigned fy = ship ? sx ^ sy : flavor == 2 ? sy : 0u;
        const unsigned f1 = role >= 4 ? fy : 0u;
        const unsigned f2 = role >= 4 ? fy : L.neg ^ ((flavor == 3 && role != 1) ? sy : 0u);
        dfac fx = dfac_of(x), fy_ = dfac_of(y);
        fx.s += L.k ^ f1; fy_.s += L.k ^ f2;
        const double s = dfac_mul0(dfac_of0(own), fx, ok), t = dfac_mul0(dfac_of0(pr), fy_, ok);
        double u = s + t;
        // 2 |X Y|, 2 X |Y| or 2 X Y
        if (role == 1) u = d_flip(s, fy);
        if (fold) {
            const unsigned sq = __shfl_sync(0xffffffffu, d_lt0(u) ? 0x80000000u : 0u, base);
            if ((role & 6) == 2) u = d_flip(u, sq);
            if (role == 0) u = d_abs(u);
        }
        const double w = u + L.g;
        return L.add ? w : u;
    }
    static __device__ __forceinline__ double coop_full(double own, double pr, double x, double y,
                                                       const Px &, const CoopLane &L, const CalcDev &C,
                                                       int role, int) {
        const int flavor = C.flavor;
        const bool ship = flavor == 1 || flavor == 5, fold = flavor >= 4;
        // coop_fast by the multiplies (nowhere ahead of their branch: computed at every
        // step they cost as much again), in one form for every role, the signs of zeros
        // and sgn(0) = 1 as in step_full (which took all six components in every
        // lane: flavor 3, 49 x 51 with a row on the axis, 1.45 -> 0.55 ms)
        const unsigned sx = d_hi(x) & 0x80000000u, sy = d_hi(y) & 0x80000000u;
        const unsigned nx = d_lt0(x) ? 0x80000000u : 0u, ny = d_lt0(y) ? 0x80000000u : 0u;
        const unsigned f1 = role < 4 ? 0u : ship ? sx ^ ny : flavor == 2 ? ny : 0u;
        const unsigned f2 = role < 4 ? L.neg ^ (flavor == 3 ? sy : 0u) : ship ? sy ^ nx : flavor == 2 ? sy : 0u;
        double fx = d_flip(x, f1);
        if (role == 1 && !ship) fx = d_mul_here(2., x);
        const double s = d_mul_here(own, fx);
        double u = d_add_here(s, d_mul_here(pr, d_flip(y, f2)));
        if (role == 1) u = ship ? fabs(s) : flavor == 2 ? d_flip(s, sy) : s;
        if (role > 1 || (role == 1 && ship)) u = d_mul_here(2., u);
        if (fold) {
            const double q = d_add_here(d_mul_here(x, x), -d_mul_here(y, y));
            if ((role & 6) == 2 && d_lt0(q)) u = -u;
            if (role == 0) u = fabs(u);
        }
        return L.add ? d_add_here(u, L.g) : u;
    }
    static __device__ __forceinline__ bool coop_near(double, double, double x, double y,
                                                     const CalcDev &C, int) {
        return d_mag_hi(cx(x, y)) >= C.esc.lo;
    }
    static __device__ __forceinline__ int coop_stop(double, double, double x, double y, const CalcDev &C,
                                                    int, int) {
        return fsg_escaped(C, cx(x, y)) ? 1 : -1;
    }
    static __device__ __forceinline__ void coop_store(double own, const Px &p, const TileDev &T, int role) {
        ((double *)T.Z)[role * ((long long)T.nx * T.ny) + p.ip] = own;
    }
    static __device__ __forceinline__ void store(const Px &p, const TileDev &T, const CalcDev &C) {
        const long long np = (long long)T.nx * T.ny, ip = p.ip;
        double *Z = (double *)T.Z;
        Z[ip] = p.X; Z[np + ip] = p.Y; Z[2 * np + ip] = p.Xa; Z[3 * np + ip] = p.Xb;
        Z[4 * np + ip] = p.Ya; Z[5 * np + ip] = p.Yb;
        if constexpr (OPT) {
            if (C.backshift > 0) {
                double xo = p.o.S.z2.x, yo = p.o.S.z2.y;
                for (int i2 = p.o.S.i2; i2 < p.n - C.backshift; i2++) {
                    double nx_, ny_;
                    bs_map(C.flavor, xo, yo, p.a, p.b, nx_, ny_);
                    xo = nx_; yo = ny_;
                }
                Z[(long long)T.i_orb * np + ip] = xo;
                Z[(long long)(T.i_orb + 1) * np + ip] = yo;
            }
        }
    }
};

template <bool OPT> __device__ __forceinline__ void std_after_step(StdPx<OPT> &p, const CalcDev &C) {
    if (p.n == 1) p.dzndz = cx(1., 0.);
}
template <bool OPT> __device__ __forceinline__ void std_after_step(StdBSPx<OPT> &, const CalcDev &) {}
template <bool OPT> __device__ __forceinline__ double2 std_z(const StdPx<OPT> &p) { return p.zn; }
template <bool OPT> __device__ __forceinline__ double2 std_z(const StdBSPx<OPT> &p) { return cx(p.X, p.Y); }

// Pixels with eight lanes each, four to a warp: `p` the pixel's state, the same
// in its lanes, where `have`.  A lane that iterates its pixel alone needs some
// 370 instructions and 1,700 clocks a step when its warp has the scheduler to
// itself, whatever the other lanes do; spread over eight lanes a step is two
// products, two FP64 sums and some eighty other instructions.  A lane with a
// factor out of range, or whose products are left open, takes the model's
// full form.
template <class Mdl>
__device__ __forceinline__ void std_coop(const WorkDev &W, const CalcDev &C, const typename Mdl::Px &p,
                                         bool have, unsigned long long &it_sum, unsigned long long &steps) {
    const int lane = threadIdx.x & 31, base = lane & ~7;
    const int role = (lane & 7) < 6 ? (lane & 7) : (lane & 7) - 6;
    const int partner = base + Mdl::coop_partner(role);
    const CoopLane L = Mdl::coop_lane(p, C, role);
    double own = have ? Mdl::coop_get(p, role) : 1.;
    int n = p.n;
    if (!__any_sync(0xffffffffu, have)) return;
    for (;;) {
        const double x = __shfl_sync(0xffffffffu, own, base), y = __shfl_sync(0xffffffffu, own, base + 1);
        const double pr = __shfl_sync(0xffffffffu, own, partner);
        int reason = -1;
        const bool near = have & Mdl::coop_near(own, pr, x, y, C, role);
        if (__any_sync(0xffffffffu, near)) {
            reason = Mdl::coop_stop(own, pr, x, y, C, base, role);
            if (n == 0) reason = -1;               // not started: nothing to test yet
        }
        if (have && reason < 0 && n + 1 >= C.max_iter) { n += 1; reason = 0; }
        if (__any_sync(0xffffffffu, have & (reason >= 0))) {
            if (have && reason >= 0) {
                const TileDev &T = W.tiles[p.t];
                if ((lane & 7) < 6) Mdl::coop_store(own, p, T, role);
                if ((lane & 7) == 0) {
                    T.stop_iter[p.ip] = n; T.stop_reason[p.ip] = (signed char)reason;
                    it_sum += (unsigned long long)n; fsg_account(W, (unsigned long long)n);
                    steps += (unsigned long long)(n - 1);
                }
                have = false;
            }
            if (!__any_sync(0xffffffffu, have)) return;
        }
        n += 1;
        bool ok = true;
        double next = Mdl::coop_fast(own, pr, x, y, L, C, base, role, ok);
        ok = ok & dfac_ok(cx(x, y)) & dfac_ok0(own) & dfac_ok0(pr);
        if (have && !ok) next = Mdl::coop_full(own, pr, x, y, p, L, C, role, n);
        if (have) own = next;
    }
}

// Up to FSG_STD_CHUNK steps of a pixel by the multiplies; its stop reason, -1 to
// go on.  Pixels on an axis and chaotic ones have zero factors or overflowing
// derivatives at every step up to max_iter, and an image's last pixels are
// such.  A warp pays for each form that one of its lanes takes, so while a lane
// is out of the integer products' range all take the multiplies.  Out of line:
// the loop keeps its registers and its instructions.  To 1000 iterations, with a
// row on the axis, Burning Ship flavor 2, 201 x 203: 1.16 ms, 1.84 with both forms
// taken, 1.40 with the multiplies alone; flavor 3 with the orbit point, 49 x 51:
// 1.10, 1.88, 1.20 ms; power 2 with d2zndc2 and the orbit point, 49 x 51: 2.12,
// 3.39, 2.64 ms (without the row: 1.13, 1.12, 2.14).  The power-2 loop without
// options has no image that this helps (its tail runs in std_coop).
template <class Mdl, bool OPT>
static __device__ __noinline__ int std_plain_chunk(typename Mdl::Px &p, const CalcDev &C) {
    typename Mdl::Px q = p;
    int reason = -1;
    for (int k = 0; k < FSG_STD_CHUNK && reason < 0; k++) {
        q.n += 1;
        reason = 0;
        if (q.n < C.max_iter) {
            Mdl::step_full(q, C);
            std_after_step<OPT>(q, C);
            reason = Mdl::stop(q, C);
        }
        std_opt_take<OPT>(q.o, C, q.n, std_z<OPT>(q));
    }
    p = q;
    return reason;
}

// The loop (core.py:2935-3056).  Pixels reach a lane in three stages:
//   * a warp claims 32 at a time and takes them through c and their first
//     steps together (a pixel lives 26 steps on the whole-set views: claimed
//     and started by its own lane, it held up the 31 others with some 25 FP64
//     instructions every step or so);
//   * they wait in the warp's part of s_px; every FSG_STD_REFILL steps the idle
//     lanes take from there;
//   * each warp runs apart until nothing is left to claim or waiting in any
//     warp of its block; from there, when at most 3/4 of the block's threads
//     hold a pixel, the states move (bit for bit) to its first
//     threads, so that the long pixels of the tail run in full warps: a warp's
//     FP64 instruction costs the pipe the same with 2 active lanes as with 32.
// The interruption flag is polled at claims and every FSG_STD_CANCEL chunks
// (numba_cycles, core.py:2959-2960); it drops the waiting pixels.
template <class Mdl, bool OPT>
__global__ void __launch_bounds__(256, OPT ? 2 : 1) k_std(WorkDev W, CalcDev C) {
    typedef typename Mdl::Px Px;
    __shared__ long long s_start[FSG_MAX_TILES_PER_LAUNCH + 1];
    __shared__ __align__(16) unsigned char s_raw[256 * sizeof(Px)];
    __shared__ int s_cnt, s_dry;
    Px *s_px = (Px *)s_raw;
    if (threadIdx.x == 0) s_dry = 0;
    fsg_load_starts(W, s_start);
    unsigned long long it_sum = 0, steps = 0;
    const int lane = threadIdx.x & 31;
    Px *queue = s_px + (threadIdx.x & ~31);
    int q_n = 0;                       // pixels waiting
    bool more = true;                  // pixels may be left to claim
    bool first = true;                 // the warp's first claim
    long long last = 0;
    Px p;
    Mdl::init(p, C, cx(0., 0.));
    bool have = false;
    const int nwarps = (int)blockDim.x >> 5;
    bool alone = true;                 // the warp runs apart from its block
    bool told = false;
    auto leave = [&](int reason) {
        const TileDev &T = W.tiles[p.t];
        Mdl::store(p, T, C);
        T.stop_iter[p.ip] = p.n; T.stop_reason[p.ip] = (signed char)reason;
        it_sum += (unsigned long long)p.n; fsg_account(W, (unsigned long long)p.n);
        steps += (unsigned long long)(p.n - 1);
        have = false;
    };
    for (int chunk = 1;; chunk++) {
        bool plain = false;
        if constexpr (Mdl::kPlain) {
            plain = __any_sync(0xffffffffu, have && !Mdl::in_range(p, C));
            if (plain) {
                Px q = p;
                const int reason = have ? std_plain_chunk<Mdl, OPT>(q, C) : -1;
                p = q;
                if (reason >= 0) leave(reason);
                __syncwarp();
            }
        }
        for (int k = plain ? FSG_STD_CHUNK : 0; k < FSG_STD_CHUNK; k++) {
            if (k % FSG_STD_REFILL == 0 && (more || q_n > 0)) {
                unsigned idle = __ballot_sync(0xffffffffu, !have);
                while (idle != 0u && (more || q_n > 0)) {
                    if (q_n == 0) {
                        Px s;
                        q_n = fsg_claim_warp(W, s_start, __popc(idle), first, last, s.t, s.ip);
                        first = false;
                        more = q_n > 0;
                        if (lane < q_n) {
                            Mdl::init(s, C, std_c(W.tiles[s.t], s.ip));
                            Mdl::start(s, C);
                            queue[lane] = s;
                        }
                        __syncwarp();
                    }
                    const int r = __popc(idle & ((1u << lane) - 1u));
                    if (!have && r < q_n) {
                        p = queue[q_n - 1 - r];
                        have = true;
                    }
                    __syncwarp();
                    q_n = max(q_n - __popc(idle), 0);
                    idle = __ballot_sync(0xffffffffu, !have);
                }
            }
            if (have) {
                p.n += 1;
                int reason;
                if (p.n >= C.max_iter) {
                    reason = 0;
                } else {
                    Mdl::step(p, C);
                    std_after_step<OPT>(p, C);
                    reason = Mdl::stop(p, C);
                }
                std_opt_take<OPT>(p.o, C, p.n, std_z<OPT>(p));
                if (reason >= 0) leave(reason);
            }
            __syncwarp();
        }
        if (alone) {
            if (chunk % FSG_STD_CANCEL == 0 && q_n > 0) {
                int stop = 0;
                if (lane == 0) stop = fsg_cancelled(W);
                if (__shfl_sync(0xffffffffu, stop, 0)) { q_n = 0; more = false; }
            }
            if (more || q_n > 0) continue;
            // dry: on alone while lanes hold pixels and another warp of the
            // block is not dry yet, then together
            int dry = 0;
            if (lane == 0) dry = told ? *(volatile int *)&s_dry : atomicAdd(&s_dry, 1) + 1;
            told = true;
            dry = __shfl_sync(0xffffffffu, dry, 0);
            if (dry < nwarps && __any_sync(0xffffffffu, have)) continue;
            alone = false;
        }
        const int live = __syncthreads_count(have);
        if (live == 0) break;
        const bool few = Mdl::kCoop && live <= 4 * nwarps;
        if (few || 4 * live <= 3 * (int)blockDim.x) {
            if (threadIdx.x == 0) s_cnt = 0;
            __syncthreads();
            if (have) s_px[atomicAdd(&s_cnt, 1)] = p;
            __syncthreads();
            if constexpr (Mdl::kCoop) {
                if (few) {
                    const int j = (int)threadIdx.x >> 3;
                    p = s_px[j < live ? j : 0];
                    std_coop<Mdl>(W, C, p, j < live, it_sum, steps);
                    break;
                }
            }
            have = (int)threadIdx.x < live;
            if (have) p = s_px[threadIdx.x];
            __syncthreads();
        }
    }
    fsg_flush_stats(W, it_sum, steps, 0ULL, 0ULL);
}

// An image of a few pixels per SM: eight lanes for each from the start
// (std_coop), no queue.  64 x 48 pixels to 200 iterations took 384 us with a
// lane per pixel.
#define FSG_STD_FEW_BLOCK 128
template <class Mdl>
__global__ void __launch_bounds__(FSG_STD_FEW_BLOCK) k_std_few(WorkDev W, CalcDev C) {
    __shared__ long long s_start[FSG_MAX_TILES_PER_LAUNCH + 1];
    fsg_load_starts(W, s_start);
    unsigned long long it_sum = 0, steps = 0;
    const long long g = W.base + blockIdx.x * (long long)(FSG_STD_FEW_BLOCK / 8) + (threadIdx.x >> 3);
    int stop = 0;
    if ((threadIdx.x & 31) == 0) stop = fsg_cancelled(W);
    const bool have = !__shfl_sync(0xffffffffu, stop, 0) && g < W.total;
    typename Mdl::Px p;
    p.t = 0; p.ip = 0;
    if (have) fsg_locate(W, s_start, g, p.t, p.ip);
    Mdl::init(p, C, have ? std_c(W.tiles[p.t], p.ip) : cx(0., 0.));
    if (have) Mdl::start(p, C);
    std_coop<Mdl>(W, C, p, have, it_sum, steps);
    fsg_flush_stats(W, it_sum, steps, 0ULL, 0ULL);
}

// Potential and distance estimate of every pixel of the launch, from the
// values the iteration kernel stored (zn, dzndc or the Jacobian, stop_iter):
// the same formulas on the same values as an in-loop epilogue, run here so
// that the lanes of a warp take them together.  Within the iteration kernel a
// pixel escapes after ~25 iterations on average and its FP64 logarithms ran
// while the other lanes of its warp waited (8.8 of 32 lanes active).
template <bool BS>
__global__ void __launch_bounds__(256) k_std_epilogue(WorkDev W, CalcDev C) {
    __shared__ long long s_start[FSG_MAX_TILES_PER_LAUNCH + 1];
    fsg_load_starts(W, s_start);
    for (long long g = W.base + blockIdx.x * (long long)blockDim.x + threadIdx.x; g < W.total;
         g += (long long)gridDim.x * blockDim.x) {
        int lo = 0, hi = W.ntiles - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_start[mid] <= g) lo = mid; else hi = mid - 1;
        }
        const TileDev &T = W.tiles[lo];
        if (T.pot == nullptr && T.dem == nullptr) continue;
        const long long ip = g - s_start[lo], np = (long long)T.nx * T.ny;
        const int n = T.stop_iter[ip];
        if (BS) {
            const double *Z = (const double *)T.Z;
            const double dXdA = Z[2 * np + ip], dXdB = Z[3 * np + ip];
            const double dYdA = Z[4 * np + ip], dYdB = Z[5 * np + ip];
            const double absd = 0.5 * (hypot(dXdA + dYdB, dXdB - dYdA) +
                                       hypot(dXdA - dYdB, dXdB + dYdA));
            fsg_epilogue(T, C, ip, cx(Z[ip], Z[np + ip]), absd, n);
        } else {
            const double2 *Z = (const double2 *)T.Z;
            const double2 d = Z[2 * np + ip];
            fsg_epilogue(T, C, ip, Z[ip], hypot(d.x, d.y), n);
        }
    }
}

// block 0: chosen by the size, CTAs of 256 under a limit on the CTAs of an SM
// (grid < 0).  Up to FSG_STD_FEW_PX pixels per SM eight lanes a pixel (no
// budget, whose claims end early); below one 256-thread CTA per SM CTAs of 64, so
// that the warps spread over the SMs.
#define FSG_STD_FEW_PX 64
template <class Mdl, bool OPT>
static void launch_k_std(const WorkDev &W, const CalcDev &C, int grid, int block, cudaStream_t s) {
    const long long total = W.total - W.base;
    if (block == 0) {
        const long long sms = fsg_auto_grid(k_std<Mdl, OPT>, -1, 256, 1LL << 40);   // one CTA per SM
        if constexpr (Mdl::kCoop) {
            if (grid == 0 && total <= FSG_STD_FEW_PX * sms && W.budget == 0 && W.order == nullptr) {
                const int per = FSG_STD_FEW_BLOCK / 8;
                k_std_few<Mdl><<<(unsigned)((total + per - 1) / per), FSG_STD_FEW_BLOCK, 0, s>>>(W, C);
                return;
            }
        }
        block = grid == 0 && total < 256 * sms ? 64 : 256;
    }
    k_std<Mdl, OPT><<<fsg_auto_grid(k_std<Mdl, OPT>, grid, block, total), block, 0, s>>>(W, C);
}

template <bool OPT>
static void launch_std(const WorkDev &W, const CalcDev &C, int grid, int block, cudaStream_t s) {
    if (C.flavor == 0 && C.nexp != 0) launch_k_std<StdMn<OPT>, OPT>(W, C, grid, block, s);
    else if (C.flavor == 0) launch_k_std<StdM2<OPT>, OPT>(W, C, grid, block, s);
    else launch_k_std<StdBS<OPT>, OPT>(W, C, grid, block, s);
    if (C.flavor == 0)
        k_std_epilogue<false><<<fsg_auto_grid(k_std_epilogue<false>, 0, 256, W.total - W.base), 256, 0, s>>>(
            W, C);
    else
        k_std_epilogue<true><<<fsg_auto_grid(k_std_epilogue<true>, 0, 256, W.total - W.base), 256, 0, s>>>(
            W, C);
}

void fsg_launch_std(const WorkDev &W, const CalcDev &C, int grid, int block, cudaStream_t s) {
    if (C.backshift > 0 || C.d2) launch_std<true>(W, C, grid, block, s);
    else launch_std<false>(W, C, grid, block, s);
}
