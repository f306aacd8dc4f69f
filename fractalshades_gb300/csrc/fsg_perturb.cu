// fsg_perturb.cu -- perturbation loops in the reference's two delta forms.
//
// Power-2 Mandelbrot: perturbation.py:988-1400 (numba_cycles_perturb,
// numba_initialize, numba_iterate) with the closures of
// models/mandelbrot_M2.py:591-627 (MN = false) or, for the power-n model,
// models/mandelbrot_Mn.py:626-733 (MN = true, fsg_mn.cuh).  XR = false is the branch with
// xr_detect_activated False (double deltas), XR = true the Xrange branch
// (double mantissa + int32 exponent, numba_xr.py semantics).
// (Burning Ship family: fsg_perturb_bs64.cu.)
//
// Built with -fmad=false so that every operation rounds once in the order of
// the reference source.  One thread iterates one pixel at a time and claims
// the next pixel from the launch's work counter as soon as it finishes.
#include "fsg_internal.cuh"

#include "fsg_bs.cuh"

__device__ __forceinline__ xc ldx(const double2 *m, const int *e, int i) {
    double2 v = __ldg(&m[i]);
    return xc_make(v.x, v.y, __ldg(&e[i]));
}

template <bool XR, bool MN, bool ORB>
__device__ __forceinline__ void pixel_m2(const TileDev &T, const CalcDev &C, long long ip,
                                         unsigned long long &nfull, unsigned long long &nbla,
                                         unsigned long long &nreb, unsigned long long &itsum) {
    const RefDev &R = *T.ref;
    const long long np = (long long)T.nx * T.ny;
    const int dzndz_on = C.interior, dzndc_on = C.calc_dzndc;
    const int order = R.order, div_iter = R.div_iter, w_wrapped = R.len;
    const int nexp = R.nexp;
    const double *Cb = R.binom;
    // perturbation.py:2214-2230 ref_path_c_from_pix, 2666-2672 lin_proj_impl
    double2 pp = fsg_pixel(T, ip);
    double px = pp.x, py = pp.y;
    double x1 = T.lin[0] * px + T.lin[1] * py;
    double y1 = T.lin[2] * px + T.lin[3] * py;
    xf dxr; dxr.m = T.dx_m; dxr.e = T.dx_e;
    xc c_xr = xr_add(xf_mul_c(dxr, cx(x1, y1)), xc_make(T.drift_re, T.drift_im, T.drift_e));
    double2 c = xr_to_std(c_xr);

    // numba_initialize :1055-1060 (the per-tile Xrange dzndz carry-over of the
    // reference is erased by the first full step, so it starts at zero here)
    double2 zn = cx(0., 0.), dzndc = cx(0., 0.), dzndz = cx(0., 0.);
    xc xzn = xc_zero(), xdzndc = xc_zero(), xdzndz = xc_zero();
    int w = 0, n = 0; signed char stop = -1;
    bool nullify = false, dyn = true;
    const xc xzero = xc_zero();
    // calc_orbit snapshots :1096-1101
    const int bs = ORB ? C.backshift : 0;
    OrbitSnap<double2> S;
    if (ORB) S.init(bs, zn);

    for (;;) {
        // BLA step :1121-1154
        if (C.bla && R.bla_len > 0 && (w & 7) == 0) {
            int ib;
            const int step = bla_possible(R, w) ? bla_lookup_z(R, zn, w, ib) : 0;
            if (step != 0) {
                double2 A = __ldg(&R.Mbla[2 * ib]), B = __ldg(&R.Mbla[2 * ib + 1]);
                n += step;
                w = (w + step) % order;
                if (XR) {
                    xzn = xr_add(xr_mul_s(A, xzn), xr_mul_s(B, c_xr));
                    zn = xr_to_std(xzn);
                    if (dzndc_on) xdzndc = xr_mul_s(A, xdzndc);
                    if (dzndz_on) xdzndz = xr_mul_s(A, xdzndz);
                } else {
                    zn = cadd(cmul(A, zn), cmul(B, c));
                    if (dzndc_on) dzndc = cmul(A, dzndc);
                    if (dzndz_on) dzndz = cmul(A, dzndz);
                }
                nbla++;
                continue;
            }
        }
        // full perturbation step :1158-1214
        n += 1;
        nfull++;
        double2 ref_zn = __ldg(&R.Zn[w]);
        xc ref_zn_xr;
        if (XR) {
            int slot = R.n_xr ? __ldg(&R.xr_slot[w]) : -1;
            ref_zn_xr = (slot >= 0) ? ldx(R.xr_m, R.xr_e, slot) : xr_from(ref_zn);
        }
        if (dzndc_on) {
            if (XR) {
                xc rd = dyn ? xzero : ldx(R.dZndc_xm, R.dZndc_xe, w);
                xdzndc = MN ? mn_p_deriv_x(nexp, Cb, xzn, xdzndc, ref_zn_xr, rd)
                            : xr_mul_2(xr_add(xr_mul(xr_add(ref_zn_xr, xzn), xdzndc), xr_mul(rd, xzn)));
            } else {
                double2 rd = dyn ? cx(0., 0.) : __ldg(&R.dZndc[w]);
                dzndc = MN ? mn_p_deriv(nexp, Cb, zn, dzndc, ref_zn, rd)
                           : rmul2(cadd(cmul(cadd(ref_zn, zn), dzndc), cmul(rd, zn)));
            }
        }
        if (dzndz_on) {
            int k = nullify ? 0 : w;
            if (XR) {
                xc rd = ldx(R.dZndz_xm, R.dZndz_xe, k);
                xdzndz = MN ? mn_p_deriv_x(nexp, Cb, xzn, xdzndz, ref_zn_xr, rd)
                            : xr_mul_2(xr_add(xr_mul(xr_add(ref_zn_xr, xzn), xdzndz), xr_mul(rd, xzn)));
            } else {
                double2 rd = __ldg(&R.dZndz[k]);
                dzndz = MN ? mn_p_deriv(nexp, Cb, zn, dzndz, ref_zn, rd)
                           : rmul2(cadd(cmul(cadd(ref_zn, zn), dzndz), cmul(rd, zn)));
            }
        }
        if (XR) {
            xzn = MN ? mn_p_zn_x(nexp, Cb, xzn, ref_zn_xr, c_xr)
                     : xr_add(xr_mul(xzn, xr_add(xzn, xr_mul_2(ref_zn_xr))), c_xr);
            zn = xr_to_std(xzn);
        } else {
            zn = MN ? mn_p_zn(nexp, Cb, zn, ref_zn, c) : cadd(cmul(zn, cadd(zn, rmul2(ref_zn))), c);
        }
        w += 1;
        if (w >= order) w = w % order;
        // max_iter :1218-1220
        if (n >= C.max_iter) { stop = 0; break; }
        // interior detection :1224-1246
        if (dzndz_on) {
            int k = nullify ? 0 : ((n == order) ? w_wrapped : w);
            bool stat;
            if (XR) {
                xc ZdZ = xr_add(xdzndz, ldx(R.dZndz_xm, R.dZndz_xe, k));
                stat = xf_sq_lt_s(xr_abs2(ZdZ), C.eps2);
            } else {
                double2 ZdZ = cadd(dzndz, __ldg(&R.dZndz[k]));
                stat = d_sq_lt(ZdZ.x * ZdZ.x + ZdZ.y * ZdZ.y, C.eps2);
            }
            if (stat) { stop = 2; break; }
        }
        // divergence :1252-1279
        double2 ref_next = __ldg(&R.Zn[w]);
        double2 ZZ = cadd(zn, ref_next);
        if (ORB) S.take(n, bs, ZZ);                                   // :1265-1273
        if (d_sq_gt(ZZ.x * ZZ.x + ZZ.y * ZZ.y, C.M2)) { stop = 1; break; }
        // rebase when the reference diverges :1283-1313
        if (w >= div_iter - 1) {
            zn = ZZ;
            if (XR) {
                xzn = xr_from(ZZ);
                if (dzndc_on) xdzndc = xr_add(xdzndc, ldx(R.dZndc_xm, R.dZndc_xe, w));
                if (dzndz_on) {
                    if (!nullify) {
                        int k = (n == order) ? w_wrapped : w;
                        xdzndz = xr_add(xdzndz, ldx(R.dZndz_xm, R.dZndz_xe, k));
                    }
                    nullify = true;
                }
            } else {
                if (dzndc_on) dzndc = cadd(dzndc, __ldg(&R.dZndc[w]));
                if (dzndz_on) {
                    if (!nullify) dzndz = cadd(dzndz, __ldg(&R.dZndz[(n == order) ? w_wrapped : w]));
                    nullify = true;
                }
            }
            w = 0; nreb++;
            continue;
        }
        // dynamic rebase :1317-1372, componentwise test
        dyn = d_abs_le(ZZ.x, zn.x) && d_abs_le(ZZ.y, zn.y);
        if (dyn) {
            if (XR) {
                int slot = R.n_xr ? __ldg(&R.xr_slot[w]) : -1;
                xc ZZx = (slot >= 0) ? xr_add(xzn, ldx(R.xr_m, R.xr_e, slot)) : xr_add_s(xzn, ref_next);
                if (xf_le(xr_abs2(ZZx), xr_abs2(xzn))) {
                    xzn = ZZx;
                    zn = xr_to_std(ZZx);
                    if (dzndc_on) xdzndc = xr_add(xdzndc, ldx(R.dZndc_xm, R.dZndc_xe, w));
                    if (dzndz_on) {
                        if (!nullify) {
                            int k = (n == order) ? w_wrapped : w;
                            xdzndz = xr_add(xdzndz, ldx(R.dZndz_xm, R.dZndz_xe, k));
                        }
                        nullify = true;
                    }
                    w = 0; nreb++;
                    continue;
                }
            } else {
                zn = ZZ;
                if (dzndc_on) dzndc = cadd(dzndc, __ldg(&R.dZndc[w]));
                if (dzndz_on) {
                    if (!nullify) dzndz = cadd(dzndz, __ldg(&R.dZndz[(n == order) ? w_wrapped : w]));
                    nullify = true;
                }
                w = 0; nreb++;
                continue;
            }
        }
    }
    // end of iterations :1375-1385
    // dzndc in the tile's unit: the reference's scale times 2^dzs
    if (XR) {
        zn = cadd(xr_to_std(xzn), __ldg(&R.Zn[w]));
        if (dzndc_on) {
            xc t = xr_add(xdzndc, ldx(R.dZndc_xm, R.dZndc_xe, w));
            t.e += T.dzs;
            dzndc = xr_to_std(t);
        }
        dzndz = cx(0., 0.);   // the Xrange branch never writes back Z[dzndz]
    } else {
        zn = cadd(zn, __ldg(&R.Zn[w]));
        if (dzndc_on) {
            dzndc = cadd(dzndc, __ldg(&R.dZndc[w]));
            if (T.dzs != 0) dzndc = cx(ldexp_d(dzndc.x, T.dzs), ldexp_d(dzndc.y, T.dzs));
        }
    }
    double2 *Z = (double2 *)T.Z;
    if (ORB) {
        // :1389-1396, the orbit point n - backshift from the full c
        double2 CC = cadd(c, __ldg(&R.Zn[1]));
        double2 zo = S.z2;
        for (int i2 = S.i2; i2 < n - bs; i2++)
            zo = MN ? cadd(mn_ipow(zo, nexp), CC) : cadd(csq(zo), CC);
        Z[(long long)T.i_orb * np + ip] = zo;
    }
    Z[ip] = zn;
    if (dzndz_on) Z[T.i_dzndz * np + ip] = dzndz;
    // Expmap: derivatives times exp(Re(ht pix) + h_moy) (perturbation.py:1387-1388)
    if (dzndc_on && T.proj) dzndc = rmul(fsg_dzndc_modifier(T, ip), dzndc);
    if (dzndc_on) Z[T.i_dzndc * np + ip] = dzndc;
    if (T.U) T.U[ip] = w;
    T.stop_iter[ip] = n;
    T.stop_reason[ip] = stop;
    fsg_epilogue(T, C, ip, zn, hypot(dzndc.x, dzndc.y), n);
    itsum += (unsigned long long)n;
}

// Whether dz = z 2^e is below half an ulp of both parts of the orbit value Z (55
// binary orders): Z + dz is then Z and dz + 2 Z is 2 Z, part by part.  False
// where a part of Z is 0 or subnormal (values held in the Xrange side table
// among them).
__device__ __forceinline__ bool dz_below(double2 Z, double2 z, int e) {
    const int lo = d_field_min(Z);
    return lo > 0 && lo - d_field_max(z) - e >= 56;
}

// The power-2 loop, both delta forms.  The reference's operations with their
// bits, arranged for GB300's pipes (an FP64 warp instruction holds its pipe for
// some 80 clocks, of which a step had 31): products on the integer pipes
// (fsg_soft.cuh), sums left out where an operand is below half an ulp of the
// other, the escape test and the BLA radii on upper words.  XR: every value is a
// mantissa and an exponent of its own frame; the bits of a value do not depend
// on the frame, so the frames of this loop differ from the reference's lazily
// normalised ones (frame_add).  Whatever leaves the ranges those forms need
// takes the reference's step, operation by operation.
template <bool XR, class Count>
__device__ __forceinline__ void pixel_m2_fast(const TileDev &T, const CalcDev &C, long long ip,
                                              Count &nfull, Count &nbla, Count &nreb, Count &itsum) {
    const RefDev &R = *T.ref;
    const long long np = (long long)T.nx * T.ny;
    const bool dzndz_on = C.interior, dzndc_on = C.calc_dzndc;
    const int order = R.order, div_iter = R.div_iter, w_wrapped = R.len;
    // perturbation.py:2214-2230 ref_path_c_from_pix, 2666-2672 lin_proj_impl
    const double2 pp = fsg_pixel(T, ip);
    const double x1 = T.lin[0] * pp.x + T.lin[1] * pp.y;
    const double y1 = T.lin[2] * pp.x + T.lin[3] * pp.y;
    xf dxr; dxr.m = T.dx_m; dxr.e = T.dx_e;
    const xc c_xr = xr_add(xf_mul_c(dxr, cx(x1, y1)), xc_make(T.drift_re, T.drift_im, T.drift_e));
    const double2 c = XR ? xm(c_xr) : xr_to_std(c_xr);
    const int ce = XR ? c_xr.e : 0;

    // dz, dz/dc, dz/dz as mantissa and exponent (FP64: exponent 0 throughout);
    // numba_initialize :1055-1060 (the per-tile Xrange dzndz carry-over of the
    // reference is erased by the first full step, so it starts at zero here)
    xc z = xc_zero(), v = xc_zero(), q = xc_zero();
    int w = 0, n = 0; signed char stop = -1;
    bool nullify = false, dyn = true;
    const xc xzero = xc_zero();
    double2 ZZ = cx(0., 0.);           // FP64: Z_w + dz of the last test,
    bool has_ZZ = false;               // when the loop came straight from it

    auto deriv_c = [&](int i) {        // dZndc_i
        return XR ? ldx(R.dZndc_xm, R.dZndc_xe, i)
                  : xc_make(__ldg(&R.dZndc[i]).x, __ldg(&R.dZndc[i]).y, 0);
    };
    auto deriv_z = [&](int i) {        // dZndz_i
        return XR ? ldx(R.dZndz_xm, R.dZndz_xe, i)
                  : xc_make(__ldg(&R.dZndz[i]).x, __ldg(&R.dZndz[i]).y, 0);
    };
    // in the ranges of the integer products: XR frames keep parts near 1, FP64
    // parts have any size
    auto ok2 = [&](double2 a, double2 b) { return XR ? dfac_ok(a) & dfac_ok(b) : cfac_ok<false>(a, b); };
    // 2 (S d + D dz) by the integer products: S (exponent eS) and dz with their
    // factors; dyn: D = 0, and S d stays as it is
    auto deriv_step = [&](double2 S, int eS, const cfac &fS, const cfac &fz, xc d, xc D, bool dyn, bool &ok) {
        ok = ok2(S, xm(d));
        const double2 a = cfac_mul(fS, cfac_of(xm(d)), ok);
        xc t = xc_make(a.x, a.y, eS + d.e);
        if (!dyn) {
            ok &= XR ? dfac_ok(xm(z)) & dfac_ok0(D.re) & dfac_ok0(D.im) : cfac_ok<true>(xm(D), xm(z));
            const double2 b = cfac_mul0(cfac_of0(xm(D)), fz, ok);
            if (XR) t = frame_add(a, eS + d.e, b, D.e + z.e, ok);
            else { t.re += b.x; t.im += b.y; }
        }
        if (XR) {
            t.e += 1;
            frame_renorm(t, ok);
        } else {
            const double2 u = rmul2(xm(t));
            t = xc_make(u.x, u.y, 0);
        }
        return t;
    };

    for (;;) {
        // BLA step :1121-1154
        if (C.bla && R.bla_len > 0 && (w & 7) == 0 && bla_possible(R, w)) {
            int ib;
            const int step = XR ? bla_lookup_x(R, z, w, ib) : bla_lookup_z(R, xm(z), w, ib);
            if (step != 0) {
                const double2 A = __ldg(&R.Mbla[2 * ib]), B = __ldg(&R.Mbla[2 * ib + 1]);
                const cfac fA = cfac_of(A);
                // A d
                auto deriv_bla = [&](xc d) {
                    bool ok = ok2(A, xm(d));
                    const double2 t = cfac_mul(fA, cfac_of(xm(d)), ok);
                    xc r = xc_make(t.x, t.y, d.e);
                    if (XR) {
                        frame_renorm(r, ok);
                        if (!ok) r = xr_mul_s(A, d);
                    } else if (!ok) {
                        const double2 u = cmul(A, xm(d));
                        r = xc_make(u.x, u.y, 0);
                    }
                    return r;
                };
                bool ok = ok2(A, xm(z)) & ok2(B, c);
                const double2 a = cfac_mul(fA, cfac_of(xm(z)), ok), b = cfac_mul(cfac_of(B), cfac_of(c), ok);
                xc nz;
                if (XR) { nz = frame_add(a, z.e, b, ce, ok); frame_renorm(nz, ok); }
                else { const double2 t = cadd(a, b); nz = xc_make(t.x, t.y, 0); }
                if (!ok) {
                    if (XR) {
                        nz = xr_add(xr_mul_s(A, z), xr_mul_s(B, c_xr));
                    } else {
                        const double2 t = cadd(cmul(A, xm(z)), cmul(B, c));
                        nz = xc_make(t.x, t.y, 0);
                    }
                }
                z = nz;
                if (dzndc_on) v = deriv_bla(v);
                if (dzndz_on) q = deriv_bla(q);
                n += step;
                w += step;
                if (w >= order) w = w % order;
                has_ZZ = false;
                nbla++;
                continue;
            }
        }
        // full perturbation step :1158-1214
        n += 1;
        nfull++;
        const double2 Z = __ldg(&R.Zn[w]);
        {
            // S = Z + dz and T2 = dz + 2 Z (exponent e2): Z and 2 Z where dz is
            // below half an ulp of Z, dz where Z is 0 (the critical point, once
            // per period)
            const bool below = dz_below(Z, xm(z), z.e);
            const bool zero = XR && d_is0(Z.x) && d_is0(Z.y) && !(R.n_xr && __ldg(&R.xr_slot[w]) >= 0);
            double2 S = Z, T2;
            int e2 = 0;
            if (XR) {
                if (zero) { S = xm(z); e2 = z.e; }
            } else if (!below) {
                if (has_ZZ) S = ZZ; else S = cadd(Z, xm(z));
            }
            T2 = S;
            if (!XR && !below) T2 = cadd(xm(z), rmul2(Z));
            const bool in = !XR | below | zero;
            const cfac fS = cfac_of(S), fz = cfac_of(xm(z));
            cfac f2 = fS;
            if (!XR && !below) f2 = cfac_of(T2);
            else if (!zero) { f2.x.s += 0x00100000u; f2.y.s += 0x00100000u; }
            xc nv = v, nq = q, nz;
            bool okz = in & ok2(T2, xm(z)), okv = true, okq = true;
            // (a derivative that is not asked for has no table to read)
            if (dzndc_on) {
                nv = deriv_step(S, e2, fS, fz, v, deriv_c(w), dyn, okv);
                okv &= in;
            }
            if (dzndz_on) {
                nq = deriv_step(S, e2, fS, fz, q, deriv_z(nullify ? 0 : w), false, okq);
                okq &= in;
            }
            const double2 p = cfac_mul(fz, f2, okz);
            if (XR) { nz = frame_add(p, e2 + z.e, c, ce, okz); frame_renorm(nz, okz); }
            else { const double2 t = cadd(p, c); nz = xc_make(t.x, t.y, 0); }
            // what is left open: the reference's operations
            if (!(okz & okv & okq)) {
                if (XR) {
                    const int slot = R.n_xr ? __ldg(&R.xr_slot[w]) : -1;
                    const xc Zx = (slot >= 0) ? ldx(R.xr_m, R.xr_e, slot) : xr_from(Z);
                    const xc S2 = xr_add(Zx, z);
                    if (!okv) nv = xr_mul_2(xr_add(xs_mul(S2, v), dyn ? xr_mul(xzero, z) : xs_mul(deriv_c(w), z)));
                    if (!okq) nq = xr_mul_2(xr_add(xs_mul(S2, q), xs_mul(deriv_z(nullify ? 0 : w), z)));
                    if (!okz) nz = xr_add(xs_mul(z, xr_add(z, xr_mul_2(Zx))), c_xr);
                } else {
                    if (!okv) {
                        const double2 D = dyn ? cx(0., 0.) : xm(deriv_c(w));
                        const double2 t = rmul2(cadd(cmul(S, xm(v)), cmul(D, xm(z))));
                        nv = xc_make(t.x, t.y, 0);
                    }
                    if (!okq) {
                        const double2 t = rmul2(cadd(cmul(S, xm(q)), cmul(xm(deriv_z(nullify ? 0 : w)), xm(z))));
                        nq = xc_make(t.x, t.y, 0);
                    }
                    if (!okz) {
                        const double2 t = cadd(cmul(xm(z), below ? rmul2(Z) : T2), c);
                        nz = xc_make(t.x, t.y, 0);
                    }
                }
            }
            z = nz; v = nv; q = nq;
        }
        w += 1;
        if (w >= order) w = w % order;
        has_ZZ = false;
        // max_iter :1218-1220
        if (n >= C.max_iter) { stop = 0; break; }
        // interior detection :1224-1246
        if (dzndz_on) {
            const xc D = deriv_z(nullify ? 0 : ((n == order) ? w_wrapped : w));
            bool stat;
            if (XR) stat = xf_sq_lt_s(xr_abs2(xr_add(q, D)), C.eps2);
            else stat = fsg_stationary(C, cadd(xm(q), xm(D)));
            if (stat) { stop = 2; break; }
        }
        const double2 Zn = __ldg(&R.Zn[w]);
        // dz below half an ulp of Z_w: Z_w + dz = Z_w, and |Z_w + dz| <= |dz| holds
        // in neither part
        if (w < div_iter - 1 && dz_below(Zn, xm(z), z.e)) {
            if (fsg_escaped(C, Zn)) { stop = 1; break; }
            dyn = false;
            ZZ = Zn;
            has_ZZ = true;
            continue;
        }
        // divergence :1252-1279
        const double2 zn = XR ? xr_to_std(z) : xm(z);
        ZZ = cadd(zn, Zn);
        if (fsg_escaped(C, ZZ)) { stop = 1; break; }
        // rebase when the reference diverges :1283-1313, dynamic rebase
        // :1317-1372 (componentwise test, in the Xrange branch confirmed on the
        // extended values)
        bool rebase = w >= div_iter - 1;
        xc nz = XR ? xr_from(ZZ) : xc_make(ZZ.x, ZZ.y, 0);
        if (!rebase) {
            dyn = d_abs_le(ZZ.x, zn.x) && d_abs_le(ZZ.y, zn.y);
            has_ZZ = !XR;
            rebase = dyn;
            if (XR && dyn) {
                const int slot = R.n_xr ? __ldg(&R.xr_slot[w]) : -1;
                nz = (slot >= 0) ? xr_add(z, ldx(R.xr_m, R.xr_e, slot)) : xr_add_s(z, Zn);
                rebase = xf_le(xr_abs2(nz), xr_abs2(z));
            }
        }
        if (rebase) {
            z = nz;
            if (dzndc_on) v = XR ? xr_add(v, deriv_c(w)) : xc_make(v.re + deriv_c(w).re, v.im + deriv_c(w).im, 0);
            if (dzndz_on) {
                if (!nullify) {
                    const xc D = deriv_z((n == order) ? w_wrapped : w);
                    q = XR ? xr_add(q, D) : xc_make(q.re + D.re, q.im + D.im, 0);
                }
                nullify = true;
            }
            w = 0; nreb++;
            has_ZZ = false;
        }
    }
    // end of iterations :1375-1385
    // dzndc in the tile's unit: the reference's scale times 2^dzs
    const double2 zn = cadd(XR ? xr_to_std(z) : xm(z), __ldg(&R.Zn[w]));
    double2 dzndc = cx(0., 0.), dzndz = cx(0., 0.);
    if (dzndc_on) {
        if (XR) {
            xc t = xr_add(v, deriv_c(w));
            t.e += T.dzs;
            dzndc = xr_to_std(t);
        } else {
            dzndc = cadd(xm(v), xm(deriv_c(w)));
            if (T.dzs != 0) dzndc = cx(ldexp_d(dzndc.x, T.dzs), ldexp_d(dzndc.y, T.dzs));
        }
    }
    // (the Xrange branch never writes back Z[dzndz])
    if (!XR) dzndz = xm(q);
    double2 *Zo = (double2 *)T.Z;
    Zo[ip] = zn;
    if (dzndz_on) Zo[T.i_dzndz * np + ip] = dzndz;
    // Expmap: derivatives times exp(Re(ht pix) + h_moy) (perturbation.py:1387-1388)
    if (dzndc_on && T.proj) dzndc = rmul(fsg_dzndc_modifier(T, ip), dzndc);
    if (dzndc_on) Zo[T.i_dzndc * np + ip] = dzndc;
    if (T.U) T.U[ip] = w;
    T.stop_iter[ip] = n;
    T.stop_reason[ip] = stop;
    fsg_epilogue(T, C, ip, zn, hypot(dzndc.x, dzndc.y), n);
    itsum += (Count)n;
}

template <bool XR, bool MN, bool ORB>
__global__ void __launch_bounds__(256) k_perturb_m2(WorkDev W, CalcDev C) {
    extern __shared__ long long s_start[];          // [W.ntiles + 1], sized at launch
    fsg_load_starts(W, s_start);
    unsigned long long nfull = 0, nbla = 0, nreb = 0, itsum = 0;
    int t; long long ip;
    while (true) {
        if (!fsg_claim_poll(W, s_start, t, ip)) break;
        const unsigned long long before = itsum;
        if constexpr (MN || ORB)
            pixel_m2<XR, MN, ORB>(W.tiles[t], C, ip, nfull, nbla, nreb, itsum);
        else
            pixel_m2_fast<XR>(W.tiles[t], C, ip, nfull, nbla, nreb, itsum);
        fsg_account(W, itsum - before);
    }
    fsg_flush_stats(W, itsum, nfull, nbla, nreb);
}

// The Xrange power-2 loop at three CTAs of 256 an SM (80 registers, with spills)
// instead of two (121): the latency of its chains bounds it.  513 x 511 pixels of
// the period-2562 nucleus take 10.0 ms so and 10.8 with two, 300 x 300 (one wave of
// three, two of two) 22 % less.  The statistics are 32-bit per pixel and summed in
// shared memory, where 64-bit sums would hold 8 registers in the loop (10.3 ms).
__global__ void __launch_bounds__(256, 3) k_perturb_m2_xr_dense(WorkDev W, CalcDev C) {
    extern __shared__ unsigned long long m2_smem[];            // sized at launch
    unsigned long long *acc = m2_smem + threadIdx.x;           // acc[k * blockDim.x]
    long long *s_start = (long long *)(m2_smem + 4 * blockDim.x);
    const int nb = blockDim.x;
    for (int k = 0; k < 4; k++) acc[k * nb] = 0ULL;
    fsg_load_starts(W, s_start);
    int t; long long ip;
    while (true) {
        if (!fsg_claim_poll(W, s_start, t, ip)) break;
        unsigned nfull = 0, nbla = 0, nreb = 0, n = 0;
        pixel_m2_fast<true>(W.tiles[t], C, ip, nfull, nbla, nreb, n);
        fsg_account(W, (unsigned long long)n);
        acc[0] += n;
        acc[nb] += nfull;
        acc[2 * nb] += nbla;
        acc[3 * nb] += nreb;
    }
    fsg_flush_stats(W, acc[0], acc[nb], acc[2 * nb], acc[3 * nb]);
}

template <bool XR, bool MN, bool ORB>
static void launch_m2(const WorkDev &W, const CalcDev &C, int grid, int block, cudaStream_t s) {
    const size_t sm = fsg_starts_smem(W);
    const long long total = W.total - W.base;
    if constexpr (XR && !MN && !ORB) {
        // Images that two CTAs an SM do not hold at once; smaller ones, and interior
        // detection, take 4 to 7 % longer with three.
        const long long two = 256LL * fsg_auto_grid(k_perturb_m2<XR, MN, ORB>, 0, 256, 1LL << 40, sm);
        if (!C.interior && total > two) {
            const size_t acc = 4 * sizeof(unsigned long long);      // per thread
            const int b = fsg_fp64_block(k_perturb_m2_xr_dense, grid, block, total, sm + 256 * acc);
            const size_t smd = sm + acc * (size_t)b;
            k_perturb_m2_xr_dense<<<fsg_auto_grid(k_perturb_m2_xr_dense, grid, b, total, smd), b, smd, s>>>(W, C);
            return;
        }
    }
    block = fsg_fp64_block(k_perturb_m2<XR, MN, ORB>, grid, block, total, sm);
    k_perturb_m2<XR, MN, ORB><<<fsg_auto_grid(k_perturb_m2<XR, MN, ORB>, grid, block, total, sm), block, sm,
                                s>>>(W, C);
}

template <bool ORB>
static void launch_m2_orb(const WorkDev &W, const CalcDev &C, int grid, int block,
                          cudaStream_t s) {
    if (C.nexp != 0 && C.mode == 1) launch_m2<true, true, ORB>(W, C, grid, block, s);
    else if (C.nexp != 0) launch_m2<false, true, ORB>(W, C, grid, block, s);
    else if (C.mode == 1) launch_m2<true, false, ORB>(W, C, grid, block, s);
    else launch_m2<false, false, ORB>(W, C, grid, block, s);
}

void fsg_launch_perturb(const WorkDev &W, const CalcDev &C, int grid, int block, cudaStream_t s) {
    if (C.flavor != 0) fsg_launch_perturb_bs(W, C, grid, block, s);
    else if (C.backshift > 0)
        launch_m2_orb<true>(W, C, grid, block, s);
    else
        launch_m2_orb<false>(W, C, grid, block, s);
}
