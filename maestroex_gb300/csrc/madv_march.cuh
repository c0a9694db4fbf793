// The PPM sweep of one column (marched) or row (by shuffles), shared by the level kernels
// (madv_march.cu) and the single-box entry points (madv_box.cu).
#pragma once
#include "madv_core.cuh"
#include "madv_exact.cuh"
#include "madv_ppm.cuh"

namespace madv {

// lanes of a warp that k_ppm_rows writes: a cell needs the slope below its low face and the
// interface value above it (ppm_type 2: positions that only pass values on, one below, two above)
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

// Ip, Im of the cells I0 .. I1 - 1 of a column (ppm_type 1); pointers at cell (low face) I0.
template <int D, int UMAC, bool INL>
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
    double um = 0, Am = 0, Bm = 0, up, Ap, Bp;
    if (UMAC) {
        um = *c.u;
        coef(um, Am, Bm);
    }
    auto none = [](int) -> double { return 0.0; };
    double s0 = ps[0], sB = ps[-st], s1 = ps[st];
    const double sA = ps[-2 * st], dA = sB - sA, d0 = s0 - sB;
    double d1 = s1 - s0;
    const double dvB = vl_slope(s0 - sA, dA, d0);
    double dv0 = vl_slope(s1 - sB, d0, d1);
    double f0 = ppm1_face_regular(sB, s0, dvB, dv0, r6);
    double sN = ps[2 * st];  // the state the next interface value needs
    for (int I = I0; I < I1; ++I) {
        const double s2 = sN;
        if (I + 1 < I1) sN = ps[3 * st];
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
        const double d2 = s2 - s1, dv1 = vl_slope(s2 - s0, d1, d2), f1 = ppm1_face_regular(s0, s1, dv0, dv1, r6);
        double sm, sp;
        if (bc.touches(I)) {
            const double2 v = ppm_cell_bnd<D, 1>(ps, st, I, bc, r6);
            sm = v.x, sp = v.y;
        } else {
            auto S = [&](int) -> double { return s0; };
            auto F = [&](int m) -> double { return m == 0 ? f0 : f1; };
            ppm_cell_any<D, 1>(S, F, none, I, 0, 0, 0, 0, sm, sp);
        }
        double ipv, imv;
        ppm_trace(s0, sm, sp, up, um, Ap, Bp, Am, Bm, epsb, ipv, imv);
        *pip = ipv;
        *pim = imv;
        pip += so;
        pim += so;
        ps += st;
        f0 = f1, dv0 = dv1, d1 = d2;
        sB = s0, s0 = s1, s1 = s2;
        um = up, Am = Ap, Bm = Bp;
    }
}

// Ip, Im of the cell i of a row (ppm_type 1), one cell a lane: slopes and interface values come from
// the neighbour lanes.  Every lane of the warp calls; the results are valid where `out`.
// Pointers at the cell (its low face).
template <int UMAC, bool INL>
__device__ __forceinline__ void ppm_row(const double* __restrict__ ps, const double* __restrict__ pu,
                                        const double* __restrict__ pA, const double* __restrict__ pB, int i, bool out,
                                        const MarchBC& bc, long long epsb, const RecipC& r6, double dt,
                                        const RecipC& rdx, double& ipv, double& imv) {
    constexpr unsigned ALL = 0xffffffffu;
    const double sB = ps[-1], s0 = ps[0], s1 = ps[1];
    const double dv = vl_slope(s1 - sB, s0 - sB, s1 - s0);
    const double dvB = __shfl_up_sync(ALL, dv, 1);
    const double f0 = ppm1_face_regular(sB, s0, dvB, dv, r6);
    const double f1 = __shfl_down_sync(ALL, f0, 1);
    if (!out) return;
    double sm, sp;
    if (bc.touches(i)) {
        const double2 v = ppm_cell_bnd<0, 1>(ps, 1, i, bc, r6);
        sm = v.x, sp = v.y;
    } else {
        auto S = [&](int) -> double { return s0; };
        auto F = [&](int m) -> double { return m == 0 ? f0 : f1; };
        auto none = [](int) -> double { return 0.0; };
        ppm_cell_any<0, 1>(S, F, none, i, 0, 0, 0, 0, sm, sp);
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

// ---- ppm_type 2, limited cells apart
// The Colella limiter changes few faces and cells -- 1-7% of the faces, 2-12% of the cells of
// the smooth fields the stage advects -- but 27-100% of the warps hold one, and its division,
// square root and curvature tests then cost the whole warp: 39-82 FP64 instructions a cell were
// issued for 20 that a lane executed.  So a warp forms the unlimited interface values of its chunk (in
// shared memory), lists the ones outside their cells and limits them 32 at a time, traces the
// cells the limiter leaves alone, lists the others and finishes those 32 at a time.
constexpr int P2_WARPS = 4;   // warps of a block
constexpr int P2_CHUNK = 21;  // cells of a column chunk at most
constexpr int P2_ROW = 512;   // positions of a row segment at most

struct P2Column {
    double f[P2_CHUNK + 3][32];
    unsigned short list[(P2_CHUNK + 3) * 32];
};
struct P2Row {
    double f[P2_ROW];
    unsigned short list[P2_ROW];
};

// lane's place in a list the warp appends to
__device__ __forceinline__ void warp_push(unsigned short* list, int& n, bool yes, int item) {
    const unsigned m = __ballot_sync(0xffffffffu, yes);
    if (yes) list[n + __popc(m & ((1u << (threadIdx.x & 31)) - 1))] = (unsigned short)item;
    n += __popc(m);
}
template <typename T>
__device__ __forceinline__ T* lane_ptr(T* p, int lane) {
    return reinterpret_cast<T*>(__shfl_sync(0xffffffffu, (unsigned long long)p, lane));
}

// A cell of the column or row: the fields at it and at its low face
struct P2Cell {
    const double *s, *u, *A, *B;
    double *ip, *im;
    int ss, su, sT;  // strides along the direction
};

// Ip, Im from the limited edge values
template <int UMAC, bool INL>
__device__ __forceinline__ void p2_trace(const P2Cell& c, double s0, double sm, double sp, double dt, const RecipC& rdx,
                                         long long epsb) {
    double up, um, Ap, Bp, Am, Bm;
    um = c.u[0];
    if (UMAC) {
        up = c.u[c.su];
        if (INL) {
            trace_coeffs(up, dt, rdx, Ap, Bp);
            trace_coeffs(um, dt, rdx, Am, Bm);
        } else {
            Ap = c.A[c.sT], Bp = c.B[c.sT], Am = c.A[0], Bm = c.B[0];
        }
    } else {
        up = um;
        if (INL) {
            trace_coeffs(up, dt, rdx, Ap, Bp);
        } else {
            Ap = c.A[0], Bp = c.B[0];
        }
        Am = Ap, Bm = Bp;
    }
    double ipv, imv;
    ppm_trace(s0, sm, sp, up, um, Ap, Bp, Am, Bm, epsb, ipv, imv);
    *c.ip = ipv;
    *c.im = imv;
}

// a listed cell of index I: the limiter in full
template <int D, int UMAC, bool INL, typename FF>
__device__ __forceinline__ void p2_limited(const P2Cell& c, FF F, int I, const MarchBC& bc, double dt, const RecipC& rdx,
                                           long long epsb, const RecipC& r6) {
    double sm, sp;
    const double* ps = c.s;
    const long st = c.ss;
    if (bc.touches(I)) {
        const double2 v = ppm_cell_bnd<D, 2>(ps, st, I, bc, r6);
        sm = v.x, sp = v.y;
    } else {
        auto S = [=](int m) -> double { return ps[m * st]; };
        auto none = [](int) -> double { return 0.0; };
        ppm_cell_any<D, 2>(S, F, none, I, 0, 0, 0, 0, sm, sp);
    }
    p2_trace<UMAC, INL>(c, *ps, sm, sp, dt, rdx, epsb);
}

// Ip, Im of the n cells from I0 of a column (n <= P2_CHUNK, 0: none; lanes may differ); c: the
// first cell.  Every lane of the warp calls.
template <int D, int UMAC, bool INL>
__device__ __forceinline__ void ppm2_column(P2Column& w, P2Cell c, int so, int I0, int n, const MarchBC& bc, double dt,
                                            const RecipC& rdx, long long epsb, const RecipC& r6) {
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int nmax = __reduce_max_sync(ALL, n);
    // interface values I0 - 1 .. I0 + n + 1
    int nl = 0;
    {
        const long st = c.ss;
        const int nf = n ? n + 3 : 0;
        const double* p = c.s;
        double a = 0, b = 0, cc = 0, d = 0;
        if (n) a = p[-3 * st], b = p[-2 * st], cc = p[-st], d = p[0];
        for (int t = 0; t < nmax + 3; ++t) {
            const bool in = t < nf;
            double nx = 0;
            if (t + 1 < nf) nx = p[(t + 1) * st];
            bool out = false;
            if (in) {
                auto S = [&](int m) -> double { return m == -2 ? a : m == -1 ? b : m == 0 ? cc : d; };
                const double se = ppm2_face_raw(S, 0);
                w.f[t][lane] = se;
                out = ppm2_face_out(se, b, cc);
            }
            warp_push(w.list, nl, out, t << 5 | lane);
            a = b, b = cc, cc = d, d = nx;
        }
    }
    __syncwarp();
    for (int q0 = 0; q0 < nl; q0 += 32) {
        const int it = w.list[min(q0 + lane, nl - 1)], ol = it & 31, t = it >> 5;
        const double* p = lane_ptr(c.s, ol);
        const long st = __shfl_sync(ALL, c.ss, ol);
        if (q0 + lane < nl) {
            p += (t - 1) * st;
            auto S = [=](int m) -> double { return p[m * st]; };
            w.f[t][ol] = ppm2_face_limit(S, 0, w.f[t][ol], r6);
        }
    }
    __syncwarp();
    // the cells the limiter leaves alone
    nl = 0;
    for (int t = 0; t < nmax; ++t) {
        bool listed = false;
        if (t < n) {
            const P2Cell x{c.s + (long)t * c.ss, c.u + (long)t * c.su, c.A + (long)t * c.sT, c.B + (long)t * c.sT,
                           c.ip + (long)t * so, c.im + (long)t * so, c.ss, c.su, c.sT};
            const double s0 = *x.s, am = w.f[t + 1][lane] - s0, ap = w.f[t + 2][lane] - s0;
            listed = bc.touches(I0 + t) || !ppm2_cell_plain(am, ap);
            if (!listed) p2_trace<UMAC, INL>(x, s0, s0 + am, s0 + ap, dt, rdx, epsb);
        }
        warp_push(w.list, nl, listed, t << 5 | lane);
    }
    __syncwarp();
    for (int q0 = 0; q0 < nl; q0 += 32) {
        const int it = w.list[min(q0 + lane, nl - 1)], ol = it & 31, t = it >> 5;
        P2Cell x;
        x.ss = __shfl_sync(ALL, c.ss, ol), x.su = __shfl_sync(ALL, c.su, ol), x.sT = __shfl_sync(ALL, c.sT, ol);
        const int o = __shfl_sync(ALL, so, ol), i0 = __shfl_sync(ALL, I0, ol);
        x.s = lane_ptr(c.s, ol) + (long)t * x.ss;
        x.u = lane_ptr(c.u, ol) + (long)t * x.su;
        x.A = lane_ptr(c.A, ol) + (long)t * x.sT;
        x.B = lane_ptr(c.B, ol) + (long)t * x.sT;
        x.ip = lane_ptr(c.ip, ol) + (long)t * o;
        x.im = lane_ptr(c.im, ol) + (long)t * o;
        if (q0 + lane < nl) {
            auto F = [&](int m) -> double { return w.f[t + 1 + m][ol]; };
            p2_limited<D, UMAC, INL>(x, F, i0 + t, bc, dt, rdx, epsb, r6);
        }
    }
}

// Ip, Im of np positions of the rows (a multiple of 32, <= P2_ROW), the first and the last two of
// which only pass interface values on.  at(p, x, i): position p's cell x and index i; false if p
// passes values on (its state is there all the same).  Every lane calls.
template <int UMAC, bool INL, typename AT>
__device__ __forceinline__ void ppm2_rows(P2Row& w, int np, AT at, const MarchBC& bc, double dt, const RecipC& rdx,
                                          long long epsb, const RecipC& r6) {
    const int lane = threadIdx.x & 31;
    int nl = 0;
    for (int p0 = 0; p0 < np; p0 += 32) {
        const int p = p0 + lane;
        P2Cell x;
        int i;
        at(p, x, i);
        const double a = x.s[-2], b = x.s[-1], cc = x.s[0], d = x.s[1];
        auto S = [&](int m) -> double { return m == -2 ? a : m == -1 ? b : m == 0 ? cc : d; };
        const double se = ppm2_face_raw(S, 0);
        w.f[p] = se;
        warp_push(w.list, nl, ppm2_face_out(se, b, cc), p);
    }
    __syncwarp();
    for (int q0 = 0; q0 < nl; q0 += 32)
        if (q0 + lane < nl) {
            const int p = w.list[q0 + lane];
            P2Cell x;
            int i;
            at(p, x, i);
            const double* ps = x.s;
            auto S = [=](int m) -> double { return ps[m]; };
            w.f[p] = ppm2_face_limit(S, 0, w.f[p], r6);
        }
    __syncwarp();
    nl = 0;
    for (int p0 = 0; p0 < np; p0 += 32) {
        const int p = p0 + lane;
        P2Cell x;
        int i;
        bool listed = false;
        if (at(p, x, i) && p >= 1 && p <= np - 3) {
            const double s0 = *x.s, am = w.f[p] - s0, ap = w.f[p + 1] - s0;
            listed = bc.touches(i) || !ppm2_cell_plain(am, ap);
            if (!listed) p2_trace<UMAC, INL>(x, s0, s0 + am, s0 + ap, dt, rdx, epsb);
        }
        warp_push(w.list, nl, listed, p);
    }
    __syncwarp();
    for (int q0 = 0; q0 < nl; q0 += 32)
        if (q0 + lane < nl) {
            const int p = w.list[q0 + lane];
            P2Cell x;
            int i;
            at(p, x, i);
            auto F = [&](int m) -> double { return w.f[p + m]; };
            p2_limited<0, UMAC, INL>(x, F, i, bc, dt, rdx, epsb, r6);
        }
}

}  // namespace madv
