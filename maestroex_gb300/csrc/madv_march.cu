// PPM and the scalar edge states with the intermediates of a direction in registers.
//
// What bounds it: FP64 issue.  One FP64 warp instruction takes the issue slots of about 64
// others on GB300 (2 FP64 lanes a clock and SM), so the FP64 instructions of the method are
// the floor, and every launch that stores an intermediate adds an index computation, its
// loads and its latency.  Three launches a direction (slopes, interfaces, cells) and twelve
// for the corner coupling of one component become six for up to three components:
//   k_ppm_march<D>  y and z: a thread marches along D over a chunk of a column, lanes along x.
//                   Every difference, slope and interface value is formed once and passed on
//                   in registers: 23 FP64 instructions a cell (ppm_type 1, counted) against 41 in
//                   three launches, one load of the state instead of nine.
//   k_ppm_rows      x: lanes along the row, slopes and interface values passed to the
//                   neighbour lane by shuffles, the warps overlapping by 2 lanes.  A march
//                   across lanes would read 32 rows at once.
//   k_ppm_march2, k_ppm_rows2  the same for ppm_type 2, the limited faces and cells listed and
//                   finished 32 at a time (madv_march.cuh): three components at 128^3 0.26 ms a
//                   direction, 0.47 ms with the limiter in place (the velocity's sweeps 0.43
//                   against 0.72 to 1.08 ms).
//   k_es_cinc       the transverse increment c_T of each cell, (dt/6/h_T) (u_T sum) times the
//                   difference of the upwind states on its T-faces: each is used by the two
//                   other directions and by both sides of a face, where the transverse
//                   kernels formed it per face.
//   k_es_trans      the six transverse states of a cell's low faces: the upwind state less the
//                   increment of its cell, one FP64 instruction each.
//   k_es_edge       the edge states of a cell's low faces from the upwind cell's four
//                   transverse states.
// The three wait on loads, not on FP64: a thread takes the faces (cells) of one direction and
// component over a chunk of a z column, so that finding its place -- five loads that wait for
// each other -- is paid once a chunk.  At 128^3 in 64^3 boxes, three components: 0.12, 0.18 and
// 0.34 ms, where the nine launches a component took 1.59 ms; one thread a face without the
// chunk 0.23, 0.26 and 0.44 ms; one thread a face that forms its own transverse states from
// the increments (one launch) 1.26 ms.  The three PPM launches: 0.80 ms against 1.67 ms.
// The arithmetic is that of the separate kernels operand by operand, so the results are
// theirs bit for bit.
#include <climits>

#include "madv_ctx.hpp"
#include "madv_exact.cuh"
#include "madv_launch.cuh"
#include "madv_march.cuh"
#include "madv_ppm.cuh"
#include "madv_slope.cuh"

namespace madv {

// ============================================================ PPM along y or z
template <int D, int UMAC>
__global__ void __launch_bounds__(256) k_ppm_march(KARGS, int fs, int sc0, int fu, int fip, int fim, unsigned lo_mask,
                                                    unsigned hi_mask, int domlo, int domhi, long long epsb, RecipC r6, unsigned nq) {
    const unsigned bx = blockIdx.x / nq, q = blockIdx.x - bx * nq;
    MADV_ELEMENT_OF(bx, R, ne, g0, g1, b, i, j, k);
    const int lo = R[e_].lo[D];
    const int I0 = lo + ((D == 1 ? j : k) - lo) * R[e_].len;
    const int I1 = min(I0 + R[e_].len, lo + R[e_].ext);
    if (D == 1) j = I0;
    else k = I0;
    const FabView s = VW(fs), ip = VW(fip + q), im = VW(fim + q), u = VW(fu), T = UMAC ? VW(F_TRA0 + D) : VW(F_TRC);
    MarchCoef c;
    c.u = &at(u, i, j, k, UMAC ? 0 : D);
    c.su = D == 1 ? u.sj : u.sk;
    c.A = &at(T, i, j, k, UMAC ? 0 : 2 * D);
    c.B = &at(T, i, j, k, UMAC ? 1 : 2 * D + 1);
    c.sT = D == 1 ? T.sj : T.sk;
    const MarchBC bc{(int)(lo_mask >> q) & 1, (int)(hi_mask >> q) & 1, domlo, domhi};
    ppm_march<D, UMAC, false>(&at(s, i, j, k, sc0 + q), D == 1 ? s.sj : s.sk, c, &at(ip, i, j, k, D),
                                    &at(im, i, j, k, D), D == 1 ? ip.sj : ip.sk, I0, I1, bc, epsb, r6);
}

// ============================================================ PPM along x
// Positions are the cells of the rows with the neighbours their interface values need; a
// warp covers 32 of them and writes the inner 30.
template <int UMAC>
__global__ void __launch_bounds__(256) k_ppm_rows(KARGS, int fs, int sc0, int fu, int fip, int fim, unsigned lo_mask,
                                                   unsigned hi_mask, int domlo, int domhi, long long epsb, RecipC r6, unsigned nq) {
    MADV_LET_NEXT();
    const unsigned bx = blockIdx.x / nq, q = blockIdx.x - bx * nq;
    const int lane = threadIdx.x & 31;
    const long w = ((long)bx * blockDim.x + threadIdx.x) >> 5;
    const long t = g0 + w * row_out(1) + lane - 1;
    const long tc = t < g0 ? g0 : (t >= g1 ? g1 - 1 : t);  // lanes past the ends work on a copy
    const int e = find_box(R, ne, tc);
    const int b = R[e].b;
    int i, j, k;
    region_ijk(R[e], tc - R[e].start, i, j, k);
    const int r = i - R[e].lo[0];
    // a cell of the row proper, not one of the lanes that only pass values on
    const bool out = t == tc && lane >= 1 && lane <= row_out(1) && r >= 1 && r <= R[e].ext;
    MADV_WAIT();
    const FabView s = VW(fs), u = VW(fu), T = UMAC ? VW(F_TRA0) : VW(F_TRC);
    const double* ps = &at(s, i, j, k, sc0 + q);
    const MarchBC bc{(int)(lo_mask >> q) & 1, (int)(hi_mask >> q) & 1, domlo, domhi};
    double ipv, imv;
    ppm_row<UMAC, false>(ps, &at(u, i, j, k, 0), &at(T, i, j, k, 0), &at(T, i, j, k, 1), i, out, bc, epsb, r6,
                               0.0, r6, ipv, imv);
    if (!out) return;
    at(VW(fip + q), i, j, k, 0) = ipv;
    at(VW(fim + q), i, j, k, 0) = imv;
}

// ============================================================ ppm_type 2
template <int D, int UMAC>
__global__ void __launch_bounds__(32 * P2_WARPS) k_ppm_march2(KARGS, int fs, int sc0, int fu, int fip, int fim,
                                                               unsigned lo_mask, unsigned hi_mask, int domlo, int domhi,
                                                               long long epsb, RecipC r6, unsigned nq) {
    __shared__ P2Column sh[P2_WARPS];
    MADV_LET_NEXT();
    const unsigned bx = blockIdx.x / nq, q = blockIdx.x - bx * nq;
    const long gid = g0 + (long)bx * blockDim.x + threadIdx.x, gc = gid < g1 ? gid : g1 - 1;
    const int e = find_box(R, ne, gc), b = R[e].b, lo = R[e].lo[D];
    int i, j, k;
    region_ijk(R[e], gc - R[e].start, i, j, k);
    const int I0 = lo + ((D == 1 ? j : k) - lo) * R[e].len, n = gid < g1 ? min(R[e].len, lo + R[e].ext - I0) : 0;
    if (D == 1) j = I0;
    else k = I0;
    MADV_WAIT();
    const FabView s = VW(fs), ip = VW(fip + q), im = VW(fim + q), u = VW(fu), T = UMAC ? VW(F_TRA0 + D) : VW(F_TRC);
    auto st = [](const FabView& f) { return D == 1 ? f.sj : (int)f.sk; };
    const P2Cell c{&at(s, i, j, k, sc0 + q), &at(u, i, j, k, UMAC ? 0 : D), &at(T, i, j, k, UMAC ? 0 : 2 * D),
                   &at(T, i, j, k, UMAC ? 1 : 2 * D + 1), &at(ip, i, j, k, D), &at(im, i, j, k, D), st(s), st(u), st(T)};
    const MarchBC bc{(int)(lo_mask >> q) & 1, (int)(hi_mask >> q) & 1, domlo, domhi};
    ppm2_column<D, UMAC, false>(sh[threadIdx.x >> 5], c, st(ip), I0, n, bc, 0.0, r6, epsb, r6);
}

template <int UMAC>
__global__ void __launch_bounds__(32 * P2_WARPS) k_ppm_rows2(KARGS, int fs, int sc0, int fu, int fip, int fim,
                                                              unsigned lo_mask, unsigned hi_mask, int domlo, int domhi,
                                                              long long epsb, RecipC r6, unsigned nq, int np) {
    __shared__ P2Row sh[P2_WARPS];
    MADV_LET_NEXT();
    const unsigned bx = blockIdx.x / nq, q = blockIdx.x - bx * nq;
    const long t0 = g0 + (((long)bx * blockDim.x + threadIdx.x) >> 5) * (np - 3) - 1;
    MADV_WAIT();
    auto at_pos = [&](int p, P2Cell& x, int& i) -> bool {
        const long t = t0 + p, tc = t < g0 ? g0 : (t >= g1 ? g1 - 1 : t);  // past the ends: a copy
        const int e = find_box(R, ne, tc), b = R[e].b;
        int j, k;
        region_ijk(R[e], tc - R[e].start, i, j, k);
        const FabView s = VW(fs), u = VW(fu), T = UMAC ? VW(F_TRA0) : VW(F_TRC);
        x = P2Cell{&at(s, i, j, k, sc0 + q), &at(u, i, j, k, 0), &at(T, i, j, k, 0), &at(T, i, j, k, 1),
                   &at(VW(fip + q), i, j, k, 0), &at(VW(fim + q), i, j, k, 0), 1, 1, 1};
        const int r = i - R[e].lo[0];
        return t == tc && r >= 1 && r <= R[e].ext;
    };
    const MarchBC bc{(int)(lo_mask >> q) & 1, (int)(hi_mask >> q) & 1, domlo, domhi};
    ppm2_rows<UMAC, false>(sh[threadIdx.x >> 5], np, at_pos, bc, 0.0, r6, epsb, r6);
}

// Cells a thread marches over: chunks short enough that the columns of the level fill the
// chip (about 2^16 threads: 430 a SM), at most 24 cells (a chunk forms two slopes and an
// interface value of its neighbour again: 2% at 24, 6% at 8 cells).
// (ppm_type 2: at most P2_CHUNK, the interface values held in shared memory.)
static int march_len(const Ctx& c) {
    long cells = 0;
    for (const HBox& v : c.ba) cells += (long)(v.hi[0] - v.lo[0] + 3) * (v.hi[1] - v.lo[1] + 3) * (v.hi[2] - v.lo[2] + 3);
    return (int)std::min(c.P.ppm_type == 2 ? (long)P2_CHUNK : 24L, std::max(2L, cells >> 16));
}

static const RegionTable& march_region(Ctx& c, int D) {
    const std::array<int, 8> key{1000, D, c.P.ppm_type, 0, 0, 0, 0, 0};
    auto it = c.regions.find(key);
    if (it != c.regions.end()) return it->second;
    RegionTable t;
    const int len = march_len(c);
    for (int b = 0; b < c.nb; ++b) {
        RegionBox r{};
        for (int d = 0; d < 3; ++d) {
            const int g = d == 2 && c.ndim == 2 ? 0 : 1;
            r.lo[d] = c.ba[b].lo[d] - g;
            r.n[d] = c.ba[b].hi[d] - c.ba[b].lo[d] + 1 + 2 * g;
        }
        r.b = b;
        r.ext = r.n[D];
        if (D == 0) {  // rows with the lanes that pass values on
            r.lo[0] -= 1;
            r.n[0] += 32 - row_out(c.P.ppm_type);
        } else {
            const int nch = (r.ext + len - 1) / len;
            r.len = (r.ext + nch - 1) / nch;
            r.n[D] = (r.ext + r.len - 1) / r.len;
        }
        r.start = t.total;
        t.total += (long)r.n[0] * r.n[1] * r.n[2];
        t.h.push_back(r);
    }
    t.d = upload_pieces(c, t.h, t.total, REGION_HINT);
    return c.regions[key] = std::move(t);
}

template <int D, int PPMT, int UMAC>
static void march_dir(Ctx& c, int fs, int sc0, int nq, const BCRecD* bc, int fu, int fip, int fim) {
    unsigned lo = 0, hi = 0;
    for (int q = 0; q < nq; ++q) {
        if (bc[q].lo[D] == BC_EXT_DIR || bc[q].lo[D] == BC_HOEXTRAP) lo |= 1u << q;
        if (bc[q].hi[D] == BC_EXT_DIR || bc[q].hi[D] == BC_HOEXTRAP) hi |= 1u << q;
    }
    const RegionTable& rt = march_region(c, D);
    const long long eb = dbits_host(c.P.rel_eps);
    const int dl = c.P.dom_lo[D], dh = c.P.dom_hi[D];
    const RecipC r6 = make_recip(6.0);
    const unsigned n = (unsigned)nq;
    if constexpr (PPMT == 2 && D == 0) {
        // positions of a warp: 512 (three components at 128^3: 0.26 ms; 0.35 at 128, where the lists
        // of a warp fill a third of a turn; 3 positions overlap the next warp), fewer where the
        // level has too few rows for 16 warps a SM
        const int np = (int)std::min((long)P2_ROW, std::max(32L, rt.total / (152 * 16) / 32 * 32));
        launch(c, rt, nq, k_ppm_rows2<UMAC>, np - 3, c.V(), fs, sc0, fu, fip, fim, lo, hi, dl, dh, eb, r6, n, np);
    } else if constexpr (PPMT == 2) {
        launch(c, rt, nq, k_ppm_march2<D, UMAC>, 0, c.V(), fs, sc0, fu, fip, fim, lo, hi, dl, dh, eb, r6, n);
    } else if constexpr (D == 0) {
        launch(c, rt, nq, k_ppm_rows<UMAC>, row_out(1), c.V(), fs, sc0, fu, fip, fim, lo, hi, dl, dh, eb, r6, n);
    } else {
        launch(c, rt, nq, k_ppm_march<D, UMAC>, 0, c.V(), fs, sc0, fu, fip, fim, lo, hi, dl, dh, eb, r6, n);
    }
}

// PPM of components sc0 .. sc0 + nq - 1 (nq <= 3) of field fs, boundary records bc[0 .. nq-1],
// into component D of fields fip + q / fim + q on the cells grown by one, for every direction
// D of dirs.  umac: traced with the face velocity fu + D (coefficients F_TRA*), else with
// component D of the cell velocity fu (coefficients F_TRC).
void ppm_march_comps(Ctx& c, int dirs, int fs, int sc0, int nq, const BCRecD* bc, int fu, int umac, int fip, int fim) {
    auto one = [&](auto dir) {
        constexpr int D = decltype(dir)::value;
        const int f = umac ? fu + D : fu;
        if (c.P.ppm_type == 1) {
            if (umac) march_dir<D, 1, 1>(c, fs, sc0, nq, bc, f, fip, fim);
            else march_dir<D, 1, 0>(c, fs, sc0, nq, bc, f, fip, fim);
        } else {
            if (umac) march_dir<D, 2, 1>(c, fs, sc0, nq, bc, f, fip, fim);
            else march_dir<D, 2, 0>(c, fs, sc0, nq, bc, f, fip, fim);
        }
    };
    if (dirs & 1) one(std::integral_constant<int, 0>{});
    if (dirs & 2) one(std::integral_constant<int, 1>{});
    if (dirs & 4) one(std::integral_constant<int, 2>{});
}

// ============================================================ ppm_type 0
// The states of MakeEdgeScalPredictor without PPM (Source/MaestroMakeEdgeScalars.cpp:662-863) kept
// per cell where PPM's Ip and Im are: above the cell s + (1 - dt u / h) / 2 slope, below it
// s - (1 + dt u / h) / 2 slope, u on the cell's high and low face.
struct SlopeBC {
    int lo[3][3], hi[3][3];  // [component][direction]
};
template <int D>
__device__ __forceinline__ void slope_state(const FabView* __restrict__ V, int nb, int b, int i, int j, int k, int sc, int q,
                                            int bclo, int bchi, int so, int dlo, int dhi, double dt, const RecipC& rh,
                                            const RecipC& r6) {
    constexpr int di = D == 0, dj = D == 1, dk = D == 2;
    const FabView s = VW(F_SOLD), u = VW(F_UMAC0 + D);
    auto S = SHIFT_S(s, sc);
    const double sl = limited_slope<D>(S, D == 0 ? i : (D == 1 ? j : k), bclo, bchi, so, dlo, dhi, r6);
    const double up = at(u, i + di, j + dj, k + dk), um = at(u, i, j, k);
    at(VW(F_IPC0 + q), i, j, k, D) = S(0) + half(1.0 - div_c(dt * up, rh)) * sl;
    at(VW(F_IMC0 + q), i, j, k, D) = S(0) - half(1.0 + div_c(dt * um, rh)) * sl;
}
__global__ void __launch_bounds__(256) k_slope_states(KARGS, int sc0, unsigned nq, SlopeBC bc, int so, int dl0, int dl1,
                                                       int dl2, int dh0, int dh1, int dh2, double dt, RecipC h0,
                                                       RecipC h1, RecipC h2, RecipC r6) {
    const unsigned bx = blockIdx.x / nq, q = blockIdx.x - bx * nq;
    MADV_ELEMENT_OF(bx, R, ne, g0, g1, b, i, j, k);
    slope_state<0>(V, nb, b, i, j, k, sc0 + q, q, bc.lo[q][0], bc.hi[q][0], so, dl0, dh0, dt, h0, r6);
    slope_state<1>(V, nb, b, i, j, k, sc0 + q, q, bc.lo[q][1], bc.hi[q][1], so, dl1, dh1, dt, h1, r6);
    slope_state<2>(V, nb, b, i, j, k, sc0 + q, q, bc.lo[q][2], bc.hi[q][2], so, dl2, dh2, dt, h2, r6);
}

void slope_states(Ctx& c, int sc0, int nq, const BCRecD* bc) {
    SlopeBC sb{};
    for (int q = 0; q < nq; ++q)
        for (int d = 0; d < 3; ++d) sb.lo[q][d] = bc[q].lo[d], sb.hi[q][d] = bc[q].hi[d];
    launch(c, rg_grow(c, 1), nq, k_slope_states, c.V(), sc0, (unsigned)nq, sb, c.P.slope_order, c.P.dom_lo[0],
           c.P.dom_lo[1], c.P.dom_lo[2], c.P.dom_hi[0], c.P.dom_hi[1], c.P.dom_hi[2], c.P.dt, make_recip(c.P.dx[0]),
           make_recip(c.P.dx[1]), make_recip(c.P.dx[2]), make_recip(6.0));
}

// ============================================================ edge states from Ip / Im
// What a face of a domain boundary does with the states on its two sides (the rules of
// MakeEdgeScalPredictor / Transverse / Edges, Source/MaestroMakeEdgeScalars.cpp:662-1667): the
// inside state whatever the velocity (foextrap, hoextrap, reflect_even), clamped to outflow
// before and after its corrections for the normal velocity component (foextrap and
// hoextrap), zero (reflect_odd), or the ghost cell's state (ext_dir).
enum { FR_UPWIND = 0, FR_INSIDE = 1, FR_CLAMP = 2, FR_ZERO = 3, FR_GHOST = 4 };
struct EsRules {
    unsigned r0, r1, r2;  // per component of the launch: 3 bits for each direction's low and high side
    // boundary faces of each direction (where no component has a rule: an index no face has)
    int lo0, lo1, lo2, hi0, hi1, hi2;
};

static EsRules es_rules(const Ctx& c, const BCRecD* bc, int comp0, int nq, int is_vel) {
    EsRules e{};
    unsigned r[3] = {0, 0, 0};
    int face[2][3];
    for (int d = 0; d < 3; ++d)
        for (int side = 0; side < 2; ++side) {
            bool any = false;
            for (int q = 0; q < nq; ++q) {
                const int t = side ? bc[q].hi[d] : bc[q].lo[d];
                unsigned code = FR_UPWIND;
                if (t == BC_EXT_DIR) code = FR_GHOST;
                else if (t == BC_REFLECT_ODD) code = FR_ZERO;
                else if (t == BC_REFLECT_EVEN) code = FR_INSIDE;
                else if (t == BC_FOEXTRAP || t == BC_HOEXTRAP) code = is_vel && comp0 + q == d ? FR_CLAMP : FR_INSIDE;
                r[q] |= code << (3 * (2 * d + side));
                any = any || code;
            }
            face[side][d] = !any ? INT_MIN : side ? c.P.dom_hi[d] + 1 : c.P.dom_lo[d];
        }
    e.r0 = r[0], e.r1 = r[1], e.r2 = r[2];
    e.lo0 = face[0][0], e.lo1 = face[0][1], e.lo2 = face[0][2];
    e.hi0 = face[1][0], e.hi1 = face[1][1], e.hi2 = face[1][2];
    return e;
}

// 0: no boundary face of direction D; 1: its low side, 2: its high side
template <int D>
__device__ __forceinline__ int face_side(const EsRules& r, int I) {
    const int lo = D == 0 ? r.lo0 : (D == 1 ? r.lo1 : r.lo2), hi = D == 0 ? r.hi0 : (D == 1 ? r.hi1 : r.hi2);
    return I == lo ? 1 : (I == hi ? 2 : 0);
}
// component q's rule on that side; bit 3: the inside cell is below the face
template <int D>
__device__ __forceinline__ unsigned face_rule(const EsRules& r, int q, int side) {
    const unsigned code = ((q == 0 ? r.r0 : q == 1 ? r.r1 : r.r2) >> (3 * (2 * D + side - 1))) & 7;
    return code ? code | (unsigned)(side - 1) << 3 : 0;
}
__device__ __forceinline__ double clamp_out(double v, bool below) { return below ? mx(v, 0.0) : mn(v, 0.0); }

// Ip, Im, the increments, the transverse states and the transverse coefficients are cell fields
// with one ghost cell: one offset serves them all.  The velocities start at the same cell.
struct EsBox {
    const double* tc;
    long s1, s2, sn;
    int lo0, lo1, lo2;
    template <int D>
    __device__ __forceinline__ long s() const { return D == 0 ? 1 : (D == 1 ? s1 : s2); }
    __device__ __forceinline__ long off(int i, int j, int k) const { return (i - lo0) + (j - lo1) * s1 + (k - lo2) * s2; }
};
__device__ __forceinline__ EsBox es_box(const FabView* __restrict__ V, int nb, int b) {
    const FabView p = VW(F_TCOEF);
    return EsBox{p.p, p.sj, p.sk, p.sn, p.lo0, p.lo1, p.lo2};
}

// The offset of one of a face's two cells: lo (below) or o.  Opaque to the compiler: the offset -1 of
// D = 0 where u < 0, folded into the address arithmetic by nvcc 13.0.88, read the wrong cell (the
// second state of a tie with u in [-rel_eps, 0), 2-way select of -1 and 0 on the sign of u).
__device__ __forceinline__ long side_offset(bool below, long lo, long o) {
    long c = below ? lo : o;
    asm("" : "+l"(c));
    return c;
}

// v less the transverse correction of the cell at o (components sn apart)
template <bool CONS>
__device__ __forceinline__ double es_less(double v, const double* c, long o, long sn) {
    return CONS ? v - c[o] - c[o + sn] + c[o + 2 * sn] : v - c[o];
}

// The state of a boundary face by its rule: of the inside one of the cells at lo (below) and o
// (above), less the increment inc of its cell (null: none).  ghost: the ext_dir state of the
// cell outside.
template <bool CONS>
__device__ __noinline__ double es_bnd(const double* ip, const double* im, const double* inc, long sn, long lo, long o,
                                      unsigned rule, const double* ghost) {
    const unsigned code = rule & 7;
    const bool below = rule & 8;
    if (code == FR_ZERO) return 0.0;
    if (code == FR_GHOST) return *ghost;
    const long oc = side_offset(below, lo, o);
    double v = (below ? ip : im)[oc];
    if (code == FR_CLAMP) v = clamp_out(v, below);
    if (inc) {
        v = es_less<CONS>(v, inc, oc, sn);
        if (code == FR_CLAMP) v = clamp_out(v, below);
    }
    return v;
}

// the state of component comp in the cell (i,j,k) + m e_d
__device__ __forceinline__ const double* es_ghost(const FabView* __restrict__ V, int nb, int b, int i, int j, int k, int d,
                                                  int m, int comp) {
    return &at(VW(F_SOLD), i + (d == 0 ? m : 0), j + (d == 1 ? m : 0), k + (d == 2 ? m : 0), comp);
}

// storage of the transverse state (A-face, corrected along B): the predictor's fields, free here
__device__ __forceinline__ int trans_field(int a, int b) {
    const int m = 2 * a + (b > a ? b - 1 : b);
    return m < 3 ? F_SL0 + m : F_SR0 + (m - 3);
}

// prologue of the three kernels: component q, direction dir, cells (i, j, k .. k1 - 1)
#define MADV_ES_COLUMN()                                                    \
    const unsigned bx_ = blockIdx.x / nq, q = blockIdx.x - bx_ * nq;        \
    MADV_PIECE(bx_, R, ne, g0, g1, b, i, j, k);                             \
    const RegionBox& r = R[e_];                                             \
    const int dir = part_, len = r.len, klo = r.lo[2], ext = r.ext;         \
    k = klo + (k - klo) * len;                                              \
    const int k1 = min(k + len, klo + ext);                                 \
    MADV_WAIT()

// The conservative form's factors: dt/3/h_T, dt/2/h_T, dt/3
struct EsCons {
    double dt3h[3], dt2h[3], dt3;
};

// c_T = F_TCOEF_T * (upwind state above - below) of the cells (F_SIMH0 + T component q holds it).
// CONS: the three terms of the correction, (dt/3/h) (s u above - s u below), (dt/3) s div u and
// (dt/3/h) s (u above - u below), in components 0, 1, 2 (one component a launch).
template <int T, bool CONS>
__device__ __forceinline__ void es_cinc(const FabView* __restrict__ V, int nb, int b, int i, int j, int k, int k1, int comp,
                                        int q, const EsRules& rules, const EsCons& ec) {
    const EsBox x = es_box(V, nb, b);
    const FabView uv = VW(F_UMAC0 + T), sv = VW(F_SOLD), dvv = VW(F_DIVU);
    const double* pu = &at(uv, i, j, k);
    const long uk = uv.sk, us = T == 0 ? 1 : (T == 1 ? uv.sj : uv.sk);
    const long o = x.off(i, j, k), s = x.s<T>();
    const double *tc = x.tc + o + T * x.sn, *ip = VW(F_IPC0 + q).p + o + T * x.sn, *im = VW(F_IMC0 + q).p + o + T * x.sn;
    double* out = VW(F_SIMH0 + T).p + o + q * x.sn;
    double um = pu[0], up = pu[us];
    for (; k < k1; ++k) {
        double un = 0, uq = 0;
        if (k + 1 < k1) {
            un = T == 2 ? up : pu[uk];
            uq = pu[uk + us];
        }
        const double t = CONS ? 0.0 : *tc;
        double vm = dhigh(um) >= 0 ? ip[-s] : im[0], vp = dhigh(up) >= 0 ? ip[0] : im[s];
        const int I = T == 0 ? i : (T == 1 ? j : k), bm = face_side<T>(rules, I), bp = face_side<T>(rules, I + 1);
        if (!nz(um)) vm = half(ip[-s] + im[0]);  // tie test |u| > 0
        if (!nz(up)) vp = half(ip[0] + im[s]);
        if (bm || bp) {
            const unsigned rm = bm ? face_rule<T>(rules, q, bm) : 0, rp = bp ? face_rule<T>(rules, q, bp) : 0;
            if (rm) vm = es_bnd<false>(ip, im, nullptr, 0, -s, 0, rm, es_ghost(V, nb, b, i, j, k, T, rm & 8 ? 0 : -1, comp));
            if (rp) vp = es_bnd<false>(ip, im, nullptr, 0, 0, s, rp, es_ghost(V, nb, b, i, j, k, T, rp & 8 ? 1 : 0, comp));
        }
        if (CONS) {
            const double s0 = at(sv, i, j, k, comp);
            out[0] = ec.dt3h[T] * (vp * up - vm * um);
            out[x.sn] = ec.dt3 * s0 * at(dvv, i, j, k);
            out[2 * x.sn] = ec.dt3h[T] * s0 * (up - um);
        } else {
            *out = t * (vp - vm);
        }
        um = un, up = uq;
        pu += uk, tc += x.s2, ip += x.s2, im += x.s2, out += x.s2;
    }
}
template <bool CONS>
__global__ void __launch_bounds__(256) k_es_cinc(KARGS, int comp0, unsigned nq, EsRules rules, EsCons ec) {
    MADV_ES_COLUMN();
    if (dir == 0) es_cinc<0, CONS>(V, nb, b, i, j, k, k1, comp0 + q, q, rules, ec);
    else if (dir == 1) es_cinc<1, CONS>(V, nb, b, i, j, k, k1, comp0 + q, q, rules, ec);
    else es_cinc<2, CONS>(V, nb, b, i, j, k, k1, comp0 + q, q, rules, ec);
}

// Transverse states of A-faces, corrected along B where the face's cells lie in the box along B
// (bi, bj: its cells in x, y; bk0 .. bk1: in z), and along C
template <int A, bool CONS>
__device__ __forceinline__ void es_trans(const FabView* __restrict__ V, int nb, int b, int i, int j, int k, int k1, bool bi,
                                         bool bj, int bk0, int bk1, int comp, int q, const EsRules& rules,
                                         long long epsb) {
    constexpr int B = A == 0 ? 1 : 0, C = A == 2 ? 1 : 2;
    const EsBox x = es_box(V, nb, b);
    const FabView uv = VW(F_UMAC0 + A);
    const double* pu = &at(uv, i, j, k);
    const long uk = uv.sk;
    const long o = x.off(i, j, k), s = x.s<A>();
    const double *ip = VW(F_IPC0 + q).p + o + A * x.sn, *im = VW(F_IMC0 + q).p + o + A * x.sn;
    const double *cb = VW(F_SIMH0 + B).p + o + q * x.sn, *cc = VW(F_SIMH0 + C).p + o + q * x.sn;
    double *qb = VW(trans_field(A, B)).p + o + q * x.sn, *qc = VW(trans_field(A, C)).p + o + q * x.sn;
    const bool wantB = B == 0 ? bi : bj;  // B is x or y
    double u = *pu;
    for (; k < k1; ++k) {
        const bool wantC = C == 1 ? bj : (k >= bk0 && k <= bk1);
        double un = 0;
        if (k + 1 < k1) un = pu[uk];
        const bool left = dhigh(u) >= 0;
        const long oc = side_offset(left, -s, 0);
        const double base = (left ? ip : im)[oc];
        double vb = 0.0, vc = 0.0;
        if (wantB) vb = es_less<CONS>(base, cb, oc, x.sn);
        if (wantC) vc = es_less<CONS>(base, cc, oc, x.sn);
        if (dmag(u) <= epsb) {  // the mean of both sides' states
            const double l = ip[-s], rr = im[0];
            if (wantB) vb = half(es_less<CONS>(l, cb, -s, x.sn) + es_less<CONS>(rr, cb, 0, x.sn));
            if (wantC) vc = half(es_less<CONS>(l, cc, -s, x.sn) + es_less<CONS>(rr, cc, 0, x.sn));
        }
        const int side = face_side<A>(rules, A == 0 ? i : (A == 1 ? j : k));
        if (side) {
            const unsigned r = face_rule<A>(rules, q, side);
            if (r) {
                const double* g = es_ghost(V, nb, b, i, j, k, A, r & 8 ? 0 : -1, comp);
                if (wantB) vb = es_bnd<CONS>(ip, im, cb, x.sn, -s, 0, r, g);
                if (wantC) vc = es_bnd<CONS>(ip, im, cc, x.sn, -s, 0, r, g);
            }
        }
        if (wantB) *qb = vb;
        if (wantC) *qc = vc;
        u = un;
        pu += uk, ip += x.s2, im += x.s2, cb += x.s2, cc += x.s2, qb += x.s2, qc += x.s2;
    }
}
template <bool CONS>
__global__ void __launch_bounds__(256) k_es_trans(KARGS, int comp0, unsigned nq, EsRules rules, long long epsb) {
    MADV_ES_COLUMN();
    // the region is grown by one across the direction: its inner cells lie in the box
    const bool bi = i > r.lo[0] && i < r.lo[0] + r.n[0] - 1, bj = j > r.lo[1] && j < r.lo[1] + r.n[1] - 1;
    const int bk0 = klo + 1, bk1 = klo + ext - 2;
    if (dir == 0) es_trans<0, CONS>(V, nb, b, i, j, k, k1, bi, bj, bk0, bk1, comp0 + q, q, rules, epsb);
    else if (dir == 1) es_trans<1, CONS>(V, nb, b, i, j, k, k1, bi, bj, bk0, bk1, comp0 + q, q, rules, epsb);
    else es_trans<2, CONS>(V, nb, b, i, j, k, k1, bi, bj, bk0, bk1, comp0 + q, q, rules, epsb);
}

// Edge states of D-faces (MakeEdgeScalEdges, Source/MaestroMakeEdgeScalars.cpp:1361-1667): what the
// faces of a column read, with pointers at the cell above the face.
template <int D, bool CONS>
struct EsFace {
    static constexpr int A = D == 0 ? 1 : 0, B = D == 2 ? 1 : 2;
    static constexpr int di = D == 0, dj = D == 1, dk = D == 2;
    const double *ip, *im, *ta, *tb, *qa, *qb, *fp, *fm;
    long s, sa, sb, s2, fs, fk;
    __device__ __forceinline__ EsFace(const FabView* __restrict__ V, int nb, int b, int i, int j, int k, int comp, int q,
                                      int force_zero, int ptf) {
        const EsBox x = es_box(V, nb, b);
        const long o = x.off(i, j, k);
        s = x.s<D>(), sa = x.s<A>(), sb = x.s<B>(), s2 = x.s2;
        ip = VW(F_IPC0 + q).p + o + D * x.sn, im = VW(F_IMC0 + q).p + o + D * x.sn;
        ta = x.tc + o + (3 + A) * x.sn, tb = x.tc + o + (3 + B) * x.sn;
        qa = VW(trans_field(A, B)).p + o + q * x.sn, qb = VW(trans_field(B, A)).p + o + q * x.sn;
        // force: the field's, or (traced) Ip of the cell below, Im of the one above
        const FabView f = VW(F_SCALFORCE);
        fs = ptf ? s : (di ? 1 : (dj ? f.sj : f.sk)), fk = ptf ? x.s2 : f.sk;
        fp = fm = nullptr;
        if (!force_zero) {
            fp = ptf ? VW(F_IPF).p + o + D * x.sn : &at(f, i, j, k, comp);
            fm = ptf ? VW(F_IMF).p + o + D * x.sn : fp;
        }
    }
    // the corrected state of the cell below the face, or above (CLAMP: and clamped at a boundary)
    template <bool CLAMP>
    __device__ __forceinline__ double state(const FabView* __restrict__ V, int nb, int b, int i, int j, int k, int comp,
                                            bool below, int force_zero, double dt2, const EsCons& ec) const {
        const long c = side_offset(below, -s, 0);
        double v = (below ? ip : im)[c];
        if (CLAMP) v = clamp_out(v, below);
        if (CONS) {
            const int m = below ? -1 : 0, ci = i + m * di, cj = j + m * dj, ck = k + m * dk;
            const FabView ua = VW(F_UMAC0 + A), ub = VW(F_UMAC0 + B), uv = VW(F_UMAC0 + D), sv = VW(F_SOLD);
            const double a0 = at(ua, ci, cj, ck), a1 = at(ua, ci + (A == 0), cj + (A == 1), ck + (A == 2));
            const double b0 = at(ub, ci, cj, ck), b1 = at(ub, ci + (B == 0), cj + (B == 1), ck + (B == 2));
            const double d0 = at(uv, ci, cj, ck), d1 = at(uv, ci + di, cj + dj, ck + dk);
            v = v - ec.dt2h[A] * (qa[c + sa] * a1 - qa[c] * a0) - ec.dt2h[B] * (qb[c + sb] * b1 - qb[c] * b0) -
                ec.dt2h[D] * at(sv, ci, cj, ck, comp) * (d1 - d0);
        } else {
            v = v - ta[c] * (qa[c + sa] - qa[c]) - tb[c] * (qb[c + sb] - qb[c]);
        }
        if (!force_zero) v = v + dt2 * (below ? fp[-fs] : fm[0]);
        if (CLAMP) v = clamp_out(v, below);
        return v;
    }
};

// a boundary face's state by its rule.  A call of its own: inlined, the clamps' four FP64
// comparisons ran on every face, where an interior one needs 6 FP64 instructions (8 with a force).
template <int D, bool CONS>
__device__ __noinline__ double es_edge_bnd(const FabView* __restrict__ V, int nb, int b, int i, int j, int k, int comp, int q,
                                           unsigned rule, int force_zero, int ptf, double dt2, const EsCons& ec) {
    const unsigned code = rule & 7;
    const bool below = rule & 8;
    if (code == FR_ZERO) return 0.0;
    if (code == FR_GHOST) return *es_ghost(V, nb, b, i, j, k, D, below ? 0 : -1, comp);
    const EsFace<D, CONS> x(V, nb, b, i, j, k, comp, q, force_zero, ptf);
    return code == FR_CLAMP ? x.template state<true>(V, nb, b, i, j, k, comp, below, force_zero, dt2, ec)
                            : x.template state<false>(V, nb, b, i, j, k, comp, below, force_zero, dt2, ec);
}

template <int D, bool CONS>
__device__ __forceinline__ void es_edge(const FabView* __restrict__ V, int nb, int b, int i, int j, int k, int k1, int comp,
                                        int oc0, int q, const EsRules& rules, int force_zero, int ptf, double dt2,
                                        long long epsb, const EsCons& ec) {
    EsFace<D, CONS> x(V, nb, b, i, j, k, comp, q, force_zero, ptf);
    const FabView uv = VW(F_UMAC0 + D), e = VW(F_SEDGE0 + D);
    const double* pu = &at(uv, i, j, k);
    const long uk = uv.sk;
    double* out = &at(e, i, j, k, oc0 + q);
    double u = *pu;
    for (; k < k1; ++k) {
        double un = 0;
        if (k + 1 < k1) un = pu[uk];
        const int side = face_side<D>(rules, D == 0 ? i : (D == 1 ? j : k));
        const unsigned r = side ? face_rule<D>(rules, q, side) : 0;
        double v;
        if (r) {
            v = es_edge_bnd<D, CONS>(V, nb, b, i, j, k, comp, q, r, force_zero, ptf, dt2, ec);
        } else {
            const bool left = dhigh(u) >= 0;
            v = x.template state<false>(V, nb, b, i, j, k, comp, left, force_zero, dt2, ec);
            if (dmag(u) <= epsb)  // the mean of both sides
                v = half(v + x.template state<false>(V, nb, b, i, j, k, comp, !left, force_zero, dt2, ec));
        }
        *out = v;
        u = un;
        pu += uk, x.ip += x.s2, x.im += x.s2, x.ta += x.s2, x.tb += x.s2, x.qa += x.s2, x.qb += x.s2;
        if (!force_zero) x.fp += x.fk, x.fm += x.fk;  // (null otherwise)
        out += e.sk;
    }
}
// Bound by the FP64 pipe (79%) with DRAM at 36%.  64 registers, four blocks an SM: 15.2 ms a 256^3
// stage at 90 registers, 12.5 at 85, 11.9 at 64; the conservative form needs its 128.
template <bool CONS>
__global__ void __launch_bounds__(256, CONS ? 2 : 4) k_es_edge(KARGS, int comp0, int oc0, unsigned nq, EsRules rules, int force_zero,
                                                  int ptf, double dt2, long long epsb, EsCons ec) {
    MADV_ES_COLUMN();
    if (dir == 0) es_edge<0, CONS>(V, nb, b, i, j, k, k1, comp0 + q, oc0, q, rules, force_zero, ptf, dt2, epsb, ec);
    else if (dir == 1) es_edge<1, CONS>(V, nb, b, i, j, k, k1, comp0 + q, oc0, q, rules, force_zero, ptf, dt2, epsb, ec);
    else es_edge<2, CONS>(V, nb, b, i, j, k, k1, comp0 + q, oc0, q, rules, force_zero, ptf, dt2, epsb, ec);
}

// Regions of the three directions one after the other (pad = D): the faces (nodal) or cells of
// direction D, grown by g across it, in z columns of at most ES_LEN cells -- shorter where the
// level has too few of them to fill the chip (about 2^19 threads).  The edge states of a 256^3 stage
// take 11.9 ms in chunks of 8, 11.6 in chunks of 16.
constexpr long ES_LEN = 16;
static const RegionTable& dirs_region(Ctx& c, bool nodal, int g) {
    const std::array<int, 8> key{1001, nodal, g, 0, 0, 0, 0, 0};
    auto it = c.regions.find(key);
    if (it != c.regions.end()) return it->second;
    RegionTable t;
    long cells = 0;
    for (const HBox& v : c.ba) cells += (long)(v.hi[0] - v.lo[0] + 1) * (v.hi[1] - v.lo[1] + 1) * (v.hi[2] - v.lo[2] + 1);
    const int len = (int)std::min(ES_LEN, std::max(1L, 3 * cells >> 19));
    for (int d = 0; d < 3; ++d)
        for (int b = 0; b < c.nb; ++b) {
            RegionBox r{};
            for (int e = 0; e < 3; ++e) {
                const int ge = e == d ? 0 : g;
                r.lo[e] = c.ba[b].lo[e] - ge;
                r.n[e] = c.ba[b].hi[e] - c.ba[b].lo[e] + 1 + 2 * ge + (e == d && nodal ? 1 : 0);
            }
            r.b = b;
            r.pad = d;
            r.ext = r.n[2];
            const int nch = (r.ext + len - 1) / len;
            r.len = (r.ext + nch - 1) / nch;
            r.n[2] = (r.ext + r.len - 1) / r.len;
            r.start = t.total;
            t.total += (long)r.n[0] * r.n[1] * r.n[2];
            t.h.push_back(r);
        }
    t.d = upload_pieces(c, t.h, t.total, REGION_HINT);
    return c.regions[key] = std::move(t);
}

// Edge states of components comp0 .. comp0 + nq - 1 (nq <= 3; conservative form: 1) of F_SOLD, 3-D,
// into components oc0 .. of F_SEDGE*: Ip / Im (slope_states, ppm_type 0) in F_IPC0 + q /
// F_IMC0 + q, the tracing and transverse coefficients of F_UMAC* or div u in place
// (edge_scal_setup).
template <bool CONS>
static void es_launch(Ctx& c, int comp0, int nq, const EsRules& r, int oc0, int force_zero) {
    const long long eb = dbits_host(c.P.rel_eps);
    const unsigned n = (unsigned)nq;
    EsCons ec{};
    ec.dt3 = c.P.dt / 3.0;
    for (int d = 0; d < 3; ++d) {
        ec.dt3h[d] = ec.dt3 / c.P.dx[d];
        ec.dt2h[d] = 0.5 * c.P.dt / c.P.dx[d];
    }
    launch(c, dirs_region(c, false, 1), nq, k_es_cinc<CONS>, c.V(), comp0, n, r, ec);
    launch(c, dirs_region(c, true, 1), nq, k_es_trans<CONS>, c.V(), comp0, n, r, eb);
    launch(c, dirs_region(c, true, 0), nq, k_es_edge<CONS>, c.V(), comp0, oc0, n, r, force_zero, c.P.ppm_trace_forces,
           0.5 * c.P.dt, eb, ec);
}
void edge_scal_ctu(Ctx& c, int comp0, int nq, const BCRecD* bc, int oc0, int force_zero, int is_vel, int is_cons) {
    const EsRules r = es_rules(c, bc, comp0, nq, is_vel);
    if (is_cons) es_launch<true>(c, comp0, nq, r, oc0, force_zero);
    else es_launch<false>(c, comp0, nq, r, oc0, force_zero);
}

}  // namespace madv
