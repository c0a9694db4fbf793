// The PPM sweep of one column (marched) or row (by shuffles), shared by the level kernels
// (madv_march.cu) and the single-box entry points (madv_box.cu).
#pragma once
#include "madv_core.cuh"
#include "madv_exact.cuh"
#include "madv_ppm.cuh"

namespace madv {

// lanes of a warp that k_ppm_rows writes: a cell needs the slope below its low face and the
// interface value above it (ppm_type 2: two above)
__host__ __device__ constexpr int row_out(int ppm_type) { return ppm_type == 1 ? 30 : 29; }

// ext_dir / hoextrap boundaries along the march
struct MarchBC {
    int lo_ext, hi_ext, domlo, domhi;
    // cells whose interface values the boundary changes
    __device__ __forceinline__ bool touches(int I) const {
        return (lo_ext && I >= domlo && I <= domlo + 2) || (hi_ext && I <= domhi && I >= domhi - 2);
    }
};

// tracing velocity and coefficients (A, B) of the first face (UMAC) or cell
struct MarchCoef {
    const double *u, *A, *B;
    long su, sT;
    double dt;    // INL: the coefficients are formed here from u
    RecipC rdx;
};

// A cell next to an ext_dir / hoextrap boundary (or in its ghost layer), everything from the
// state: few cells, kept out of line.
template <int D, int PPMT>
__device__ __noinline__ double2 ppm_cell_bnd(const double* ps, long st, int I, MarchBC bc, RecipC r6) {
    auto S = [=](int m) -> double { return ps[m * st]; };
    auto DV = [=](int m) -> double { return vl_at(S, m); };
    auto F = [=](int m) -> double {
        return ppm_face_any<PPMT>(S, DV, m, I + m, bc.lo_ext, bc.hi_ext, bc.domlo, bc.domhi, r6);
    };
    auto FR = [=](int m) -> double {
        return PPMT == 2 ? ppm2_face_regular(S, m, r6) : ppm1_face_regular(S(m - 1), S(m), DV(m - 1), DV(m), r6);
    };
    double2 v;
    ppm_cell_any<D, PPMT>(S, F, FR, I, bc.lo_ext, bc.hi_ext, bc.domlo, bc.domhi, v.x, v.y);
    return v;
}

// Ip, Im of the cells I0 .. I1 - 1 of a column; pointers at cell (low face) I0.
template <int D, int PPMT, int UMAC, bool INL>
__device__ __forceinline__ void ppm_march(const double* __restrict__ ps, long st, MarchCoef c, double* __restrict__ pip,
                                          double* __restrict__ pim, long so, int I0, int I1, const MarchBC& bc,
                                          long long epsb, const RecipC& r6) {
    auto coef = [&](double u, double& A, double& B) {
        if (INL) {
            trace_coeffs(u, c.dt, c.rdx, A, B);
        } else {
            A = *c.A;
            B = *c.B;
        }
    };
    double um, Am, Bm, up, Ap, Bp;
    if (UMAC) {
        um = *c.u;
        coef(um, Am, Bm);
    }
    double s0 = ps[0], sB = ps[-st], s1 = ps[st];
    double d1 = s1 - s0;
    double dv0 = 0, f0 = 0, fm = 0, f1 = 0, sA = 0, s2 = 0;
    auto none = [](int) -> double { return 0.0; };
    if (PPMT == 1) {
        const double sa = ps[-2 * st], dA = sB - sa, d0 = s0 - sB;
        const double dvB = vl_slope(s0 - sa, dA, d0);
        dv0 = vl_slope(s1 - sB, d0, d1);
        f0 = ppm1_face_regular(sB, s0, dvB, dv0, r6);
    } else {
        sA = ps[-2 * st];
        s2 = ps[2 * st];
        auto S = [&](int m) -> double {
            return m == -3 ? ps[-3 * st] : m == -2 ? sA : m == -1 ? sB : m == 0 ? s0 : m == 1 ? s1 : s2;
        };
        fm = ppm2_face_regular(S, -1, r6);
        f0 = ppm2_face_regular(S, 0, r6);
        f1 = ppm2_face_regular(S, 1, r6);
    }
    constexpr int AHEAD = PPMT == 1 ? 2 : 3;
    double sN = ps[AHEAD * st];  // the state the next interface value needs
    for (int I = I0; I < I1; ++I) {
        const double snext = sN;
        if (I + 1 < I1) sN = ps[(AHEAD + 1) * st];
        if (UMAC) {
            c.u += c.su;
            c.A += c.sT;
            c.B += c.sT;
        }
        up = *c.u;
        coef(up, Ap, Bp);
        if (!UMAC) {
            um = up, Am = Ap, Bm = Bp;
            c.u += c.su;
            c.A += c.sT;
            c.B += c.sT;
        }
        double sm, sp, f2 = 0, dv1 = 0, d2 = 0;
        if (PPMT == 1) {
            d2 = snext - s1;
            dv1 = vl_slope(snext - s0, d1, d2);
            f1 = ppm1_face_regular(s0, s1, dv0, dv1, r6);
        } else {
            auto S = [&](int m) -> double { return m == 0 ? s0 : m == 1 ? s1 : m == 2 ? s2 : snext; };
            f2 = ppm2_face_regular(S, 2, r6);
        }
        if (bc.touches(I)) {
            const double2 v = ppm_cell_bnd<D, PPMT>(ps, st, I, bc, r6);
            sm = v.x, sp = v.y;
        } else {
            auto S = [&](int m) -> double { return m == -2 ? sA : m == -1 ? sB : m == 0 ? s0 : m == 1 ? s1 : s2; };
            auto F = [&](int m) -> double { return m == -1 ? fm : m == 0 ? f0 : m == 1 ? f1 : f2; };
            ppm_cell_any<D, PPMT>(S, F, none, I, 0, 0, 0, 0, sm, sp);
        }
        double ipv, imv;
        ppm_trace(s0, sm, sp, up, um, Ap, Bp, Am, Bm, epsb, ipv, imv);
        *pip = ipv;
        *pim = imv;
        pip += so;
        pim += so;
        ps += st;
        if (PPMT == 2) {
            sA = sB, fm = f0, f0 = f1, f1 = f2;
            sB = s0, s0 = s1, s1 = s2, s2 = snext;
        } else {
            f0 = f1, dv0 = dv1, d1 = d2;
            sB = s0, s0 = s1, s1 = snext;
        }
        um = up, Am = Ap, Bm = Bp;
    }
}

// Ip, Im of the cell i of a row, one cell a lane: slopes and interface values come from the
// neighbour lanes.  Every lane of the warp calls; the results are valid where `out`.
// Pointers at the cell (its low face).
template <int PPMT, int UMAC, bool INL>
__device__ __forceinline__ void ppm_row(const double* __restrict__ ps, const double* __restrict__ pu,
                                        const double* __restrict__ pA, const double* __restrict__ pB, int i, bool out,
                                        const MarchBC& bc, long long epsb, const RecipC& r6, double dt,
                                        const RecipC& rdx, double& ipv, double& imv) {
    constexpr unsigned ALL = 0xffffffffu;
    const double sB = ps[-1], s0 = ps[0], s1 = ps[1];
    double fm = 0, f0, f1, f2 = 0;
    if (PPMT == 1) {
        const double dv = vl_slope(s1 - sB, s0 - sB, s1 - s0);
        const double dvB = __shfl_up_sync(ALL, dv, 1);
        f0 = ppm1_face_regular(sB, s0, dvB, dv, r6);
        f1 = __shfl_down_sync(ALL, f0, 1);
    } else {
        const double sA = ps[-2];
        auto S = [&](int m) -> double { return m == -2 ? sA : m == -1 ? sB : m == 0 ? s0 : s1; };
        f0 = ppm2_face_regular(S, 0, r6);
        fm = __shfl_up_sync(ALL, f0, 1);
        f1 = __shfl_down_sync(ALL, f0, 1);
        f2 = __shfl_down_sync(ALL, f0, 2);
    }
    if (!out) return;
    double sm, sp;
    if (bc.touches(i)) {
        const double2 v = ppm_cell_bnd<0, PPMT>(ps, 1, i, bc, r6);
        sm = v.x, sp = v.y;
    } else {
        auto S = [&](int m) -> double { return m == 0 ? s0 : m == -1 ? sB : m == 1 ? s1 : ps[m]; };
        auto F = [&](int m) -> double { return m == -1 ? fm : m == 0 ? f0 : m == 1 ? f1 : f2; };
        auto none = [](int) -> double { return 0.0; };
        ppm_cell_any<0, PPMT>(S, F, none, i, 0, 0, 0, 0, sm, sp);
    }
    double up, um, Ap, Bp, Am, Bm;
    if (UMAC) {
        up = pu[1], um = pu[0];
        if (INL) {
            trace_coeffs(up, dt, rdx, Ap, Bp);
            trace_coeffs(um, dt, rdx, Am, Bm);
        } else {
            Ap = pA[1], Bp = pB[1], Am = pA[0], Bm = pB[0];
        }
    } else {
        up = um = pu[0];
        if (INL) {
            trace_coeffs(up, dt, rdx, Ap, Bp);
        } else {
            Ap = pA[0], Bp = pB[0];
        }
        Am = Ap, Bm = Bp;
    }
    ppm_trace(s0, sm, sp, up, um, Ap, Bp, Am, Bm, epsb, ipv, imv);
}

}  // namespace madv
