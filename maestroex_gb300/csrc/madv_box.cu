// Single-box entry points: Maestro::PPM on one box (Source/Maestro.H:1396,
// Source/MaestroPPM.cpp:5-2262), the routine the reference calls once per box and per
// traced component.
//
// One launch: the blocks are divided among the three directions, each running the sweep of
// the level kernels (madv_march.cuh: columns marched along y and z, rows by shuffles, ppm_type
// 2's limited cells listed) with the tracing coefficients formed where they are used.  No
// scratch.  Twelve dependent launches with every intermediate in memory spent their time
// between launches: 63 us a call for a 34^3 box, 28 us now (17 us on the device, the rest the
// caller's side and the launch).
#include "madv_ctx.hpp"
#include "madv_exact.cuh"
#include "madv_launch.cuh"
#include "madv_march.cuh"

namespace madv {

struct PPMBoxArgs {
    FabView s, u[3], ip, im;
    RecipC rdx[3], r6;
    MarchBC bc[3];
    RegionBox r[3];   // x: rows with the lanes that pass values on; y, z: columns in chunks
    long total[3];    // threads (x: positions)
    unsigned first[3];  // first block of each direction
    int sc, np;
    long long epsb;
    double dt;
};

template <int D>
__device__ __forceinline__ int stride_of(const FabView& f) { return D == 0 ? 1 : (D == 1 ? f.sj : (int)f.sk); }

template <int D, int PPMT, int UMAC>
__device__ __forceinline__ void box_column(const PPMBoxArgs& a, P2Column* sh) {
    const long t = (long)(blockIdx.x - a.first[D]) * blockDim.x + threadIdx.x;
    const bool in = t < a.total[D];
    int i, j, k;
    region_ijk(a.r[D], in ? t : a.total[D] - 1, i, j, k);
    const int lo = a.r[D].lo[D], I0 = lo + ((D == 1 ? j : k) - lo) * a.r[D].len, I1 = min(I0 + a.r[D].len, lo + a.r[D].ext);
    if (D == 1) j = I0;
    else k = I0;
    const FabView u = a.u[D];
    const double* pu = &at(u, i, j, k);
    double *ip = &at(a.ip, i, j, k, D), *im = &at(a.im, i, j, k, D);
    const double* ps = &at(a.s, i, j, k, a.sc);
    if (PPMT == 1) {
        if (!in) return;
        MarchCoef c;
        c.u = pu, c.A = c.B = pu;
        c.su = stride_of<D>(u), c.sT = 0;
        c.dt = a.dt, c.rdx = a.rdx[D];
        ppm_march<D, UMAC, true>(ps, stride_of<D>(a.s), c, ip, im, stride_of<D>(a.ip), I0, I1, a.bc[D], a.epsb, a.r6);
    } else {
        const P2Cell c{ps, pu, pu, pu, ip, im, stride_of<D>(a.s), stride_of<D>(u), 0};
        ppm2_column<D, UMAC, true>(sh[threadIdx.x >> 5], c, stride_of<D>(a.ip), I0, in ? I1 - I0 : 0, a.bc[D], a.dt,
                                   a.rdx[D], a.epsb, a.r6);
    }
}

template <int UMAC>
__device__ __forceinline__ void box_rows1(const PPMBoxArgs& a) {
    const int lane = threadIdx.x & 31;
    const long w = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long t = w * row_out(1) + lane - 1, tc = t < 0 ? 0 : (t >= a.total[0] ? a.total[0] - 1 : t);
    int i, j, k;
    region_ijk(a.r[0], tc, i, j, k);
    const int r = i - a.r[0].lo[0];
    const bool out = t == tc && lane >= 1 && lane <= row_out(1) && r >= 1 && r <= a.r[0].ext;
    const double* pu = &at(a.u[0], i, j, k);
    double ip, im;
    ppm_row<UMAC, true>(&at(a.s, i, j, k, a.sc), pu, pu, pu, i, out, a.bc[0], a.epsb, a.r6, a.dt, a.rdx[0], ip, im);
    if (!out) return;
    at(a.ip, i, j, k, 0) = ip;
    at(a.im, i, j, k, 0) = im;
}

template <int UMAC>
__device__ __forceinline__ void box_rows2(const PPMBoxArgs& a, P2Row* sh) {
    const long t0 = (((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (a.np - 3) - 1;
    auto at_pos = [&](int p, P2Cell& x, int& i) -> bool {
        const long t = t0 + p, tc = t < 0 ? 0 : (t >= a.total[0] ? a.total[0] - 1 : t);
        int j, k;
        region_ijk(a.r[0], tc, i, j, k);
        const double* pu = &at(a.u[0], i, j, k);
        x = P2Cell{&at(a.s, i, j, k, a.sc), pu, pu, pu, &at(a.ip, i, j, k, 0), &at(a.im, i, j, k, 0), 1, 1, 0};
        const int r = i - a.r[0].lo[0];
        return t == tc && r >= 1 && r <= a.r[0].ext;
    };
    ppm2_rows<UMAC, true>(sh[threadIdx.x >> 5], a.np, at_pos, a.bc[0], a.dt, a.rdx[0], a.epsb, a.r6);
}

constexpr int BOX_TPB = 32 * P2_WARPS;

template <int PPMT, int UMAC>
__global__ void __launch_bounds__(BOX_TPB) k_ppm_box(PPMBoxArgs a) {
    __shared__ union Sh {
        P2Column c[PPMT == 2 ? P2_WARPS : 1];
        P2Row r[PPMT == 2 ? P2_WARPS : 1];
    } sh;
    MADV_LET_NEXT();
    MADV_WAIT();
    if (blockIdx.x >= a.first[2]) box_column<2, PPMT, UMAC>(a, sh.c);
    else if (blockIdx.x >= a.first[1]) box_column<1, PPMT, UMAC>(a, sh.c);
    else if (PPMT == 1) box_rows1<UMAC>(a);
    else box_rows2<UMAC>(a, sh.r);
}

static FabView view_of(const madv_fab& f) {
    FabView v{};
    v.p = f.p;
    v.lo0 = f.lo[0];
    v.lo1 = f.lo[1];
    v.lo2 = f.lo[2];
    const long nx = f.hi[0] - f.lo[0] + 1, ny = f.hi[1] - f.lo[1] + 1, nz = f.hi[2] - f.lo[2] + 1;
    v.sj = (int)nx;
    v.sk = nx * ny;
    v.sn = nx * ny * nz;
    return v;
}

static bool covers(const madv_fab* f, const int lo[3], const int hi[3], int ncomp) {
    if (!f || !f->p || f->ncomp < ncomp) return false;
    for (int d = 0; d < 3; ++d)
        if (f->lo[d] > lo[d] || f->hi[d] < hi[d]) return false;
    return true;
}

// Validates the arguments and runs the PPM of one box.  Returns a madv error code.
int ppm_box_run(const madv_params& P, const madv_box* bx, const madv_fab* s, int comp, const madv_fab* u,
                const madv_fab* v, const madv_fab* w, int is_umac, const int* bc, const madv_fab* Ip,
                const madv_fab* Im, cudaStream_t st, long& launches) {
    if (!bx || !s || !u || !v || !w || !bc || !Ip || !Im) return MADV_ERR_PARAM;
    if (P.ppm_type != 1 && P.ppm_type != 2) {
        set_error("madv_ppm: ppm_type must be 1 or 2 (ppm_type 0 uses the slopes)");
        return MADV_ERR_UNSUPPORTED;
    }
    int n[3];
    for (int d = 0; d < 3; ++d) {
        n[d] = bx->hi[d] - bx->lo[d] + 1;
        if (n[d] <= 0) return MADV_ERR_LAYOUT;
    }
    const int g = P.ppm_type == 2 ? 3 : 2;
    int slo[3], shi[3];
    for (int d = 0; d < 3; ++d) {
        slo[d] = bx->lo[d] - g;
        shi[d] = bx->hi[d] + g;
    }
    if (!covers(s, slo, shi, comp + 1)) {
        set_error("madv_ppm: s must cover the box grown by 2 (ppm_type 1) or 3 (ppm_type 2) ghost cells");
        return MADV_ERR_LAYOUT;
    }
    const madv_fab* vel[3] = {u, v, w};
    for (int d = 0; d < 3; ++d) {
        int hi[3] = {bx->hi[0], bx->hi[1], bx->hi[2]};
        if (is_umac) hi[d] += 1;
        if (!covers(vel[d], bx->lo, hi, 1)) {
            set_error("madv_ppm: tracing velocity FAB does not cover the box (faces if is_umac)");
            return MADV_ERR_LAYOUT;
        }
    }
    if (!covers(Ip, bx->lo, bx->hi, 3) || !covers(Im, bx->lo, bx->hi, 3)) {
        set_error("madv_ppm: Ip/Im must be 3-component FABs covering the box");
        return MADV_ERR_LAYOUT;
    }
    PPMBoxArgs a{};
    a.s = view_of(*s);
    a.sc = comp;
    a.ip = view_of(*Ip);
    a.im = view_of(*Im);
    a.epsb = dbits_host(P.rel_eps);
    a.dt = P.dt;
    a.r6 = make_recip(6.0);
    const long cells = (long)n[0] * n[1] * n[2];
    // chunks of a column short enough for 2^14 threads a direction; a box this small is bound by
    // latency, and the two slopes and the interface value a chunk repeats cost nothing
    const int len = (int)std::min((long)P2_CHUNK, std::max(2L, cells >> 14));
    unsigned blocks = 0;
    for (int d = 0; d < 3; ++d) {
        a.bc[d] = MarchBC{bc[d] == BC_EXT_DIR || bc[d] == BC_HOEXTRAP, bc[3 + d] == BC_EXT_DIR || bc[3 + d] == BC_HOEXTRAP,
                          P.dom_lo[d], P.dom_hi[d]};
        a.rdx[d] = make_recip(P.dx[d]);
        a.u[d] = view_of(*vel[d]);
        RegionBox& r = a.r[d];
        for (int e = 0; e < 3; ++e) {
            r.lo[e] = bx->lo[e];
            r.n[e] = n[e];
        }
        r.ext = n[d];
        if (d == 0) {
            r.lo[0] -= 1;
            r.n[0] += 32 - row_out(P.ppm_type);
        } else {
            const int nch = (n[d] + len - 1) / len;
            r.len = (n[d] + nch - 1) / nch;
            r.n[d] = (n[d] + r.len - 1) / r.len;
        }
        r.dv = piece_div(r.n);
        a.total[d] = (long)r.n[0] * r.n[1] * r.n[2];
        a.first[d] = blocks;
        long threads = a.total[d];
        if (d == 0) {
            a.np = (int)std::min((long)P2_ROW, std::max(32L, a.total[0] / (152 * 8) / 32 * 32));
            const int out = P.ppm_type == 1 ? row_out(1) : a.np - 3;
            threads = (a.total[0] + out - 1) / out * 32;
        }
        blocks += (unsigned)((threads + BOX_TPB - 1) / BOX_TPB);
    }
    void (*kern)(PPMBoxArgs) = P.ppm_type == 1 ? (is_umac ? k_ppm_box<1, 1> : k_ppm_box<1, 0>)
                                               : (is_umac ? k_ppm_box<2, 1> : k_ppm_box<2, 0>);
    launch_on(st, false, dim3(blocks), BOX_TPB, kern, a);
    ++launches;
    return cuda_ok(cudaGetLastError(), "madv_ppm launch") ? MADV_OK : MADV_ERR_CUDA;
}

}  // namespace madv
