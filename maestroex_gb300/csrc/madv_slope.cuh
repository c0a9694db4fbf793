// Limited slopes for ppm_type 0 (Maestro::Slopex/y/z, Source/MaestroSlopes.cpp:6-600), one
// cell of index I along D, S(m) the field m cells along D.
#pragma once
#include "madv_ppm.cuh"

namespace madv {

template <int D, typename SF>
__device__ __forceinline__ double limited_slope(SF S, int I, int bclo, int bchi, int slope_order, int ilo, int ihi,
                                                const RecipC& r6) {
    const bool lo_ext = (bclo == BC_EXT_DIR || bclo == BC_HOEXTRAP);
    const bool hi_ext = (bchi == BC_EXT_DIR || bchi == BC_HOEXTRAP);
    double out = 0.0;
    if (slope_order == 2) {
        double del = half(S(1) - S(-1));
        double dpls = 2.0 * (S(1) - S(0));
        double dmin = 2.0 * (S(0) - S(-1));
        double slim = mn(fabs(dpls), fabs(dmin));
        slim = dpls * dmin > 0.0 ? slim : 0.0;
        double sflag = copysign(1.0, del);
        out = sflag * mn(slim, fabs(del));
        if (lo_ext) {
            if (I == ilo - 1) {
                out = 0.0;
            } else if (I == ilo) {
                del = (S(1) + 3.0 * S(0) - 4.0 * S(-1)) / 3.0;
                dpls = 2.0 * (S(1) - S(0));
                dmin = 2.0 * (S(0) - S(-1));
                slim = mn(fabs(dpls), fabs(dmin));
                slim = dpls * dmin > 0.0 ? slim : 0.0;
                sflag = copysign(1.0, del);
                out = sflag * mn(slim, fabs(del));
            }
        }
        if (hi_ext) {
            if (I == ihi + 1) {
                out = 0.0;
            } else if (I == ihi) {
                del = -(S(-1) + 3.0 * S(0) - 4.0 * S(1)) / 3.0;
                dpls = 2.0 * (S(0) - S(-1));
                dmin = 2.0 * (S(1) - S(0));
                slim = mn(fabs(dpls), fabs(dmin));
                slim = dpls * dmin > 0.0 ? slim : 0.0;
                sflag = copysign(1.0, del);
                out = sflag * mn(slim, fabs(del));
            }
        }
    } else if (slope_order == 4) {
        // dcen, dmin, dpls of the three cells and their limited slopes dxl, dxr; the
        // differences are formed once, the limits on the integer pipe (vl_slope).  A NaN among the
        // cells makes a difference NaN: the comparisons then give slope 0 where the product of
        // two differences is NaN, and pass a NaN ds on.
        const double e0 = S(-1) - S(-2), e1 = S(0) - S(-1), e2 = S(1) - S(0), e3 = S(2) - S(1);
        const bool n0 = is_nan(e0), n1 = is_nan(e1), n2 = is_nan(e2), n3 = is_nan(e3);
        double dxl = n0 || n1 ? 0.0 : vl_slope(S(0) - S(-2), e0, e1), dxr = n2 || n3 ? 0.0 : vl_slope(S(2) - S(0), e2, e3);
        const double dcen = half(S(1) - S(-1));
        double dmin = twice(e1), dpls = twice(e2);
        const double dlim = !n1 && !n2 && prod_gt0(dpls, dmin) ? __longlong_as_double(min(dmag(dmin), dmag(dpls))) : 0.0;
        double ds = 4.0 / 3.0 * dcen - div_6(dxr + dxl, r6);
        auto limited = [&](double v) {  // copysign(1, dcen) * min(|v|, dlim)
            return is_nan(v) ? v : dsigned(__longlong_as_double(min(dmag(v), dmag(dlim))), dcen);
        };
        out = limited(ds);
        // the x sweep tests the centred dlim where y and z test the one-sided slim
        if (lo_ext) {
            if (I == ilo - 1) {
                out = 0.0;
            } else if (I == ilo) {
                double del = -16.0 / 15.0 * S(-1) + 0.5 * S(0) + 2.0 / 3.0 * S(1) - 0.1 * S(2);
                dmin = 2.0 * (S(0) - S(-1));
                dpls = 2.0 * (S(1) - S(0));
                double slim = mn(fabs(dpls), fabs(dmin));
                slim = dpls * dmin > 0.0 ? (D == 0 ? dlim : slim) : 0.0;
                double sflag = copysign(1.0, del);
                out = sflag * mn(slim, fabs(del));
            } else if (I == ilo + 1) {
                double del = -16.0 / 15.0 * S(-2) + 0.5 * S(-1) + 2.0 / 3.0 * S(0) - 0.1 * S(1);
                dmin = 2.0 * (S(-1) - S(-2));
                dpls = 2.0 * (S(0) - S(-1));
                double slim = mn(fabs(dpls), fabs(dmin));
                slim = dpls * dmin > 0.0 ? (D == 0 ? dlim : slim) : 0.0;
                double sflag = copysign(1.0, del);
                dxl = sflag * mn(slim, fabs(del));
                ds = 4.0 / 3.0 * dcen - (dxr + dxl) / 6.0;
                out = limited(ds);
            }
        }
        if (hi_ext) {
            if (I == ihi + 1) {
                out = 0.0;
            } else if (I == ihi) {
                double del = -(-16.0 / 15.0 * S(1) + 0.5 * S(0) + 2.0 / 3.0 * S(-1) - 0.1 * S(-2));
                dmin = 2.0 * (S(0) - S(-1));
                dpls = 2.0 * (S(1) - S(0));
                double slim = mn(fabs(dpls), fabs(dmin));
                slim = dpls * dmin > 0.0 ? (D == 0 ? dlim : slim) : 0.0;
                double sflag = copysign(1.0, del);
                out = sflag * mn(slim, fabs(del));
            } else if (I == ihi - 1) {
                double del = -(-16.0 / 15.0 * S(2) + 0.5 * S(1) + 2.0 / 3.0 * S(0) - 0.1 * S(-1));
                dmin = 2.0 * (S(1) - S(0));
                dpls = 2.0 * (S(2) - S(1));
                double slim = mn(fabs(dpls), fabs(dmin));
                slim = dpls * dmin > 0.0 ? (D == 0 ? dlim : slim) : 0.0;
                double sflag = copysign(1.0, del);
                dxr = sflag * mn(slim, fabs(del));
                ds = 4.0 / 3.0 * dcen - (dxl + dxr) / 6.0;
                out = limited(ds);
            }
        }
    }
    return out;
}

}  // namespace madv
