// Per-element PPM arithmetic shared by the level kernels (madv_kernels.cu) and the
// single-box entry points (madv_box.cu).  Source: Maestro::PPM,
// Source/MaestroPPM.cpp (ppm_type 1 x-sweep :33-252, ppm_type 2 x-sweep :254-771; the y and
// z sweeps :779-2260 are the same algorithm with the differences kept as flags below).
#pragma once
#include "madv_core.cuh"
#include "madv_exact.cuh"

namespace madv {

// S(m): the field at cell (index + m) along direction D.
#define SHIFT_S(s, sc) [&](int m) -> double { return at(s, i + m * di, j + m * dj, k + m * dk, sc); }

// Van Leer slope from the differences c = s(1) - s(-1), l = s(0) - s(-1), r = s(1) - s(0)
// (Source/MaestroPPM.cpp:37-73): dsc = c/2, dsl = 2l, dsr = 2r, and if (dsl*dsr > 0)
// copysign(1, dsc) * min(|dsc|, min(|dsl|, |dsr|)).  The minimum of non-negative (finite)
// doubles is the minimum of their bit patterns, and copysign(1, dsc) * m with m >= 0 is m
// with the sign of dsc.  No FP64 instruction.
__device__ __forceinline__ double vl_slope(double c, double l, double r) {
    const double dsl = twice(l), dsr = twice(r);
    if (!prod_gt0(dsl, dsr)) return 0.0;
    return dsigned(__longlong_as_double(min(dmag(half(c)), min(dmag(dsl), dmag(dsr)))), c);
}

// Van Leer slope of cell (i,j,k) along D (Source/MaestroPPM.cpp:37-73).
template <int D>
__device__ __forceinline__ double ppm_dsvl(const FabView& s, int sc, int i, int j, int k) {
    constexpr int di = D == 0, dj = D == 1, dk = D == 2;
    auto S = SHIFT_S(s, sc);
    return vl_slope(S(1) - S(-1), S(0) - S(-1), S(1) - S(0));
}

// Fourth-order interface value (ppm_type 2) of the face between cells m-1 and m of S, S(q) the
// field q cells along D, before it is limited.
template <typename SF>
__device__ __forceinline__ double ppm2_face_raw(SF S, int m) {
    return (7.0 / 12.0) * (S(m - 1) + S(m)) - (1.0 / 12.0) * (S(m - 2) + S(m + 1));
}
// Whether it may lie outside its two cells a, b.  reference: (se - s(m-1)) * (s(m) - se) < 0, i.e.
// the product of (se - s(m-1)) and -(s(m) - se) = se - s(m) (exact) is positive.  The
// differences have the sign of the comparison (on integer keys, no FP64 instruction) unless se
// is infinite or NaN, whose differences may be NaN: ppm2_face_limit decides on those.
__device__ __forceinline__ bool ppm2_face_out(double se, double a, double b) {
    const long long ks = dkey(se), ka = dkey(a), kb = dkey(b);
    return (ks > ka && ks > kb) || (ks < ka && ks < kb) || (dhigh(se) & 0x7ff00000) == 0x7ff00000;
}
// Colella's limited curvature max(min(a, 1.25 min of the signed curvatures), 0), a >= 0, as
// mx(mn(..), 0) of FP64 comparisons gives it.  Finite ones: the smallest positive curvature by its
// bit pattern (x -> RN(1.25 x) keeps the order), 0 where one is not positive -- one FP64
// instruction instead of six or eight.
__device__ __forceinline__ bool all_finite(double a, double b, double c) {
    return max(max(dmag(a), dmag(b)), dmag(c)) < 0x7ff0000000000000LL;
}
__device__ __forceinline__ double limited_curvature(double a, double fl, double fr) {
    const double C = 1.25;
    if (!all_finite(a, fl, fr)) return mx(mn(C * fl, mn(C * fr, a)), 0.0);
    const long long m = min(dbits(fl), dbits(fr));
    if (m <= 0) {
        // the comparisons' zero: -0 where the first of the smallest is one
        const bool mz = !nz(fl) ? dbits(fl) < 0 : dbits(fr) < 0;
        return lt0(fl) || lt0(fr) || !mz ? 0.0 : -0.0;
    }
    return __longlong_as_double(min(dbits(C * __longlong_as_double(m)), dbits(a)));
}

// the limited value of one that does
template <typename SF>
__device__ __forceinline__ double ppm2_face_limit(SF S, int m, double se, const RecipC& r6) {
    if (prod_gt0(se - S(m - 1), se - S(m))) {
        double D2 = 3.0 * (S(m - 1) - twice(se) + S(m));
        double D2L = S(m - 2) - twice(S(m - 1)) + S(m);
        double D2R = S(m - 1) - twice(S(m)) + S(m + 1);
        const bool neg = dhigh(D2) < 0;  // sgn = copysign(1, D2): sgn * x is x or -x
        double D2LIM = dflip(limited_curvature(dabs(D2), dflip(D2L, neg), dflip(D2R, neg)), neg);
        se = half(S(m - 1) + S(m)) - div_6(D2LIM, r6);
    }
    return se;
}
// Interior fourth-order limited face value (ppm_type 2).
template <typename SF>
__device__ __forceinline__ double ppm2_face_regular(SF S, int m, const RecipC& r6) {
    const double se = ppm2_face_raw(S, m);
    return ppm2_face_out(se, S(m - 1), S(m)) ? ppm2_face_limit(S, m, se, r6) : se;
}
// Whether the cell limiter leaves alpham = f0 - s0, alphap = f1 - s0 as they are: neither an
// extremum (alpham * alphap >= 0) nor one more than twice the other.
__device__ __forceinline__ bool ppm2_cell_plain(double alpham, double alphap) {
    return prod_gt0(alpham, dflip(alphap)) && !(dmag(alphap) > dmag(twice(alpham))) &&
           !(dmag(alpham) > dmag(twice(alphap)));
}

// Van Leer slope of the cell m of S, and the interior interface value between cells m-1 and m
// (ppm_type 1).
template <typename SF>
__device__ __forceinline__ double vl_at(SF S, int m) {
    return vl_slope(S(m + 1) - S(m - 1), S(m) - S(m - 1), S(m + 1) - S(m));
}
__device__ __forceinline__ double ppm1_face_regular(double sl, double sr, double dvl, double dvr, const RecipC& r6) {
    return clamp_between(half(sr + sl) - div_6(dvr - dvl, r6), sr, sl);
}

// Limited interface value of the face of index f along D, between cells m-1 and m of S
// (ppm_type 1 :37-111, ppm_type 2 :257-335; the boundary stencils of :131-205 / :443-700
// are the values the reference assigns to the faces next to an ext_dir/hoextrap
// boundary).  DV(m): van Leer slope of cell m (ppm_type 1).
template <int PPMT, typename SF, typename DF>
__device__ __forceinline__ double ppm_face_any(SF S, DF DV, int m, int f, int lo_ext, int hi_ext, int domlo, int domhi,
                                               const RecipC& r6) {
    double v;
    if (lo_ext && f == domlo) {
        v = S(m - 1);
    } else if (hi_ext && f == domhi + 1) {
        v = S(m);
    } else if (lo_ext && f == domlo + 1) {
        v = -0.2 * S(m - 2) + 0.75 * S(m - 1) + 0.5 * S(m) - 0.05 * S(m + 1);
        v = mx(v, mn(S(m), S(m - 1)));
        v = mn(v, mx(S(m), S(m - 1)));
    } else if (hi_ext && f == domhi) {
        v = -0.2 * S(m + 1) + 0.75 * S(m) + 0.5 * S(m - 1) - 0.05 * S(m - 2);
        v = mx(v, mn(S(m - 1), S(m)));
        v = mn(v, mx(S(m - 1), S(m)));
    } else if (PPMT == 1) {
        v = ppm1_face_regular(S(m - 1), S(m), DV(m - 1), DV(m), r6);
    } else {
        v = ppm2_face_regular(S, m, r6);
    }
    return v;
}

// The same for the face (i,j,k) of a field with its van Leer slopes stored per cell.
template <int D, int PPMT>
__device__ __forceinline__ double ppm_face_value(const FabView& s, int sc, const FabView& dv, int i, int j, int k,
                                                 int lo_ext, int hi_ext, int domlo, int domhi, const RecipC& r6) {
    constexpr int di = D == 0, dj = D == 1, dk = D == 2;
    auto S = SHIFT_S(s, sc);
    auto DV = SHIFT_S(dv, 0);
    return ppm_face_any<PPMT>(S, DV, 0, D == 0 ? i : (D == 1 ? j : k), lo_ext, hi_ext, domlo, domhi, r6);
}

// Characteristic-tracing coefficients (Source/MaestroPPM.cpp:209-251):
// sigma = |u| dt / dx, A = 0.5 sigma, B = 1 - 2/3 sigma.
__device__ __forceinline__ void trace_coeffs(double u, double dt, const RecipC& rdx, double& A, double& B) {
    const double sigma = div_c(dabs(u) * dt, rdx);
    A = half(sigma);
    B = 1.0 - 2.0 / 3.0 * sigma;
}

__device__ __forceinline__ bool finite2(double a, double b) {
    return (dhigh(a) & 0x7ff00000) != 0x7ff00000 && (dhigh(b) & 0x7ff00000) != 0x7ff00000;
}

// Edge values sm, sp of the cell of index I along D from the face values F (quadratic limiter
// :117-128 for ppm_type 1, Colella-2008 limiter :337-434 for ppm_type 2, with the
// boundary re-limiting of :131-205 / :443-700).  S(m): the field m cells along D; F(m): the
// interface value between cells m-1 and m.
//
// F holds, on the two faces next to an ext_dir/hoextrap boundary, the values the reference
// assigns for the first interior cells.  Cells outside the domain (ghost cells of a grown
// box) are not re-limited by the reference and see the regular interpolants on those faces,
// FR(m).
template <int D, int PPMT, typename SF, typename FF, typename RF>
__device__ __forceinline__ void ppm_cell_any(SF S, FF F, RF FR, int I, int lo_ext, int hi_ext, int domlo, int domhi,
                                             double& sm, double& sp) {
    const bool outside = (lo_ext && I < domlo) || (hi_ext && I > domhi);
    auto Fc = [&](int m) -> double {
        const int f = I + m;
        if (outside && ((lo_ext && (f == domlo || f == domlo + 1)) || (hi_ext && (f == domhi || f == domhi + 1))))
            return FR(m);
        return F(m);
    };
    const double s0 = S(0);
    if (PPMT == 1) {
        sm = Fc(0);
        sp = Fc(1);
        const bool special = (lo_ext && I == domlo) || (hi_ext && I == domhi);
        if (!special) {
            // reference: (sp-s0)*(s0-sm) <= 0;  |sp-s0| >= 2|sm-s0|;  |sm-s0| >= 2|sp-s0|.
            // sm-s0 = -(s0-sm) exactly; non-negative doubles compare like their bit patterns.
            const double a = sp - s0, q = s0 - sm;
            const long long ma = dmag(a), mq = dmag(q);
            if (!prod_gt0(a, q)) {
                sp = s0;
                sm = s0;
            } else {
                // the two cases as one expression, so that a warp with both issues it once
                const bool up = ma >= dmag(twice(q)), dn = mq >= dmag(twice(a));
                if (up || dn) {
                    const double v = 3.0 * s0 - twice(up ? sm : sp);
                    if (up) sp = v;
                    else sm = v;
                }
            }
        }
    } else {
        double sedgel = Fc(-1), sedge = Fc(0), sedger = Fc(1), sedgerr = Fc(2);
        if (D == 0 && hi_ext && I == domhi - 1) sedgerr = FR(2);
        if (lo_ext && I == domlo) {
            sm = sedge;
            sp = sedger;
        } else if (hi_ext && I == domhi) {
            sp = sedger;
            sm = sedge;
        } else {
            const double bigm_tol = (D == 0 && lo_ext && (I == domlo + 1 || I == domlo + 2)) ? 1.e10 : 1.e-10;
            double alphap = sedger - s0;
            double alpham = sedge - s0;
            // |alphap| > 2|alpham| and |alpham| > 2|alphap| on magnitudes' bit patterns;
            // alpham * alphap >= 0 is "not (alpham * -alphap > 0)"
            const long long mp = dmag(alphap), mm = dmag(alpham);
            const bool bigp = mp > dmag(twice(alpham));
            const bool bigm = mm > dmag(twice(alphap));
            bool extremum = false;
            if (!prod_gt0(alpham, dflip(alphap))) {
                extremum = true;
            } else if (bigp || bigm) {
                double dafacem = sedge - sedgel;
                double dafacep = sedgerr - sedger;
                double dabarm = s0 - S(-1);
                double dabarp = S(1) - s0;
                // (the minimum of a pair is NaN where its first value is, and no minimum compares then)
                const bool face = !is_nan(dafacem) && !is_nan(dabarm) &&
                                  min(dmag(dafacem), dmag(dafacep)) >= min(dmag(dabarm), dmag(dabarp));
                extremum = !prod_gt0(face ? dafacem : dabarm, face ? dafacep : dabarp);
            }
            if (extremum) {
                double D2 = 6.0 * (alpham + alphap);
                double D2L = S(-2) - twice(S(-1)) + s0;
                double D2R = s0 - twice(S(1)) + S(2);
                double D2C = S(-1) - twice(s0) + S(1);
                const bool neg = dhigh(D2) < 0;  // sgn = copysign(1, D2)
                const double fl = dflip(D2L, neg), fr = dflip(D2R, neg), fc = dflip(D2C, neg), a = dabs(D2);
                const double C = 1.25;
                double D2LIM;
                if (all_finite(fl, fr, fc) && dmag(a) < 0x7ff0000000000000LL) {
                    const long long m = min(min(dbits(fl), dbits(fr)), dbits(fc));
                    D2LIM = m <= 0 ? 0.0 : __longlong_as_double(min(dbits(C * __longlong_as_double(m)), dbits(a)));
                } else {
                    D2LIM = mx(mn(a, mn(C * fl, mn(C * fr, C * fc))), 0.0);
                }
                if (nz(D2LIM) || !finite2(alpham, alphap)) {
                    // one divisor: its reciprocal, then 4 FP64 instructions a quotient
                    const RecipV r = recip_v(mx(a, 1.e-10));
                    alpham = div_v(alpham * D2LIM, r);
                    alphap = div_v(alphap * D2LIM, r);
                } else {  // a finite alpha times 0 over a positive number: the zero of its sign
                    alpham = dsigned(0.0, alpham);
                    alphap = dsigned(0.0, alphap);
                }
            } else {
                // |alphap| > 2|alpham| and |alpham| > 2|alphap| exclude each other: the two
                // one-sided rewrites as one, on (a, b) = (alpham, alphap) or (alphap, alpham), so
                // that a warp with both issues the division and the square root once
                if (bigp || bigm) {
                    const double a = bigp ? alpham : alphap, b = bigp ? alphap : alpham;
                    const bool neg = dhigh(a) < 0;  // sgn = copysign(1, a)
                    const double tol = bigp ? 1.e-10 : bigm_tol;
                    const double amax = dflip(b) * b / twice(twice(alpham + alphap));
                    const double del = (bigp ? S(-1) : S(1)) - s0;
                    if (dflip(amax, neg) >= dflip(del, neg)) {
                        double v = dflip(twice(a));
                        if (dflip(del - a, neg) >= tol)
                            v = dflip(twice(del)) - dflip(twice(sqrt(del * del - del * a)), neg);
                        if (bigp) alphap = v;
                        else alpham = v;
                    }
                }
            }
            sm = s0 + alpham;
            sp = s0 + alphap;
        }
    }
}

// The same for cell (i,j,k) of a field with stored interface values F and slopes dv.
template <int D, int PPMT>
__device__ __forceinline__ void ppm_cell_edges(const FabView& s, int sc, const FabView& F, const FabView& dv, int i,
                                               int j, int k, int lo_ext, int hi_ext, int domlo, int domhi,
                                               const RecipC& r6, double& sm, double& sp) {
    constexpr int di = D == 0, dj = D == 1, dk = D == 2;
    auto S = SHIFT_S(s, sc);
    auto FS = SHIFT_S(F, 0);
    auto DV = SHIFT_S(dv, 0);
    auto FR = [&](int m) -> double {
        return PPMT == 2 ? ppm2_face_regular(S, m, r6) : ppm1_face_regular(S(m - 1), S(m), DV(m - 1), DV(m), r6);
    };
    ppm_cell_any<D, PPMT>(S, FS, FR, D == 0 ? i : (D == 1 ? j : k), lo_ext, hi_ext, domlo, domhi, sm, sp);
}

__device__ __forceinline__ double trace_side(double sm, double sp, double d, double s6, double A, double B, bool p) {
    return (p ? sp : sm) + dflip(A * (d + dflip(B * s6, p)), p);
}

// Characteristic tracing of one cell: Ip from the velocity at the high face (coefficients
// Ap, Bp), Im from the low face (Am, Bm); tb = bits(rel_eps).
__device__ __forceinline__ void ppm_trace(double s0, double sm, double sp, double up, double um, double Ap, double Bp,
                                          double Am, double Bm, long long tb, double& ip, double& im) {
    // ip = sp - Ap (sp - sm - Bp s6) where up > rel_eps, im = sm + Am (sp - sm + Bm s6) where
    // um < -rel_eps; x - y is x + (-y), so both are one expression up to signs, issued once
    // for a warp whose lanes need the one or the other (a cell that needs both -- flow out
    // through both faces -- takes a second turn)
    ip = s0;
    im = s0;
    const bool p = gt_t(up, tb), m = lt_negt(um, tb);
    if (!p && !m) return;
    const double s6 = 6.0 * s0 - 3.0 * (sm + sp), d = sp - sm;
    const double v = trace_side(sm, sp, d, s6, p ? Ap : Am, p ? Bp : Bm, p);
    if (p) ip = v;
    else im = v;
    if (p && m) im = trace_side(sm, sp, d, s6, Am, Bm, false);
}

}  // namespace madv
