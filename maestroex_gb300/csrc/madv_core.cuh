// Device-side building blocks of the scalar-advection stage.
//
// Data layout in HBM: every field of a level is one allocation holding one FAB per box
// (the box grown by the field's ghost width, nodal in the face direction for face data),
// Fortran order (i fastest) and one contiguous block per component, i.e. the
// amrex::FArrayBox layout the reference's Array4 views index.  A kernel sees a field
// through a FabView per box.
//
// Work decomposition: a launch covers one index region per box (e.g. the box grown by one
// cell, or its nodal x-faces).  The regions of all boxes are laid end to end; thread gid
// finds its box from a hint table (the piece of every 128th element, behind the pieces) and
// its cell by multiplications with precomputed reciprocals of the extents, so one launch
// covers boxes of any (uneven) sizes.  A binary search of the prefix and 64-bit divisions
// took 200 of the 300 instructions a thread of the small kernels issued, and a chain of
// dependent loads as long as the search is deep.  The per-box form of a launch restricts [g0, g1) to one box.
#pragma once
#include <cstdint>

namespace madv {

// AMReX BCType / PhysBCType values used by the reference.
enum { BC_REFLECT_ODD = -1, BC_INT_DIR = 0, BC_REFLECT_EVEN = 1, BC_FOEXTRAP = 2,
       BC_EXT_DIR = 3, BC_HOEXTRAP = 4 };
enum { PB_INTERIOR = 0, PB_INFLOW = 1, PB_OUTFLOW = 2, PB_SYMMETRY = 3, PB_SLIPWALL = 4,
       PB_NOSLIPWALL = 5 };
enum { RHO = 0, RHOH = 1, TEMP = 2, PI = 3, FIRSTSPEC = 4 };

constexpr int MAX_SCAL = 64;

struct FabView {
    double* p;  // element (lo) of component 0
    int lo0, lo1, lo2;
    int sj;
    long sk, sn;
};

__host__ __device__ __forceinline__ double& at(const FabView& f, int i, int j, int k, int n = 0) {
    return f.p[(long)(i - f.lo0) + (long)(j - f.lo1) * f.sj + (long)(k - f.lo2) * f.sk + (long)n * f.sn];
}

// l / n and l / (n m) for l < 2^31 by multiplication: with s = ceil(log2 n) and
// m = ceil(2^(31+s) / n) < 2^32 the quotient is (l m) >> (31+s), exact because
// l (m n - 2^(31+s)) < 2^31 2^s (Granlund and Montgomery, PLDI 1994).  m = 0: n is 1.
// sh[0] = -2: a piece of 2^31 elements or more, divided in 64 bits.
struct PieceDiv {
    unsigned m[2];
    int sh[2];
};

struct RegionBox {
    int lo[3];
    int n[3];
    int b;  // box owning this piece of the region
    int pad;
    long start;
    PieceDiv dv;
    int ext, len;  // march regions: cells along the march, and of one chunk
};

__host__ __device__ inline PieceDiv piece_div(const int* n) {
    PieceDiv v{};
    if ((double)n[0] * n[1] * n[2] >= 2147483648.0) {
        v.sh[0] = -2;
        return v;
    }
    for (int d = 0; d < 2; ++d) {
        int s = 0;
        while ((1LL << s) < n[d]) ++s;
        v.m[d] = n[d] == 1 ? 0u : (unsigned)(((1ULL << (31 + s)) + n[d] - 1) / n[d]);
        v.sh[d] = s - 1;  // after the high word of the product
    }
    return v;
}

struct BCRecD {
    int lo[3];
    int hi[3];
};

// The piece owning element gid: the pieces are followed by one whose start is the total and
// by the hint table, the piece of every (1 << SH)th element.
constexpr int REGION_HINT = 7, COPY_HINT = 5;
template <int SH, typename Piece>
__device__ __forceinline__ int find_piece(const Piece* __restrict__ R, int ne, long gid) {
    if (ne == 1) return 0;
    const int* __restrict__ hint = reinterpret_cast<const int*>(R + ne + 1);
    int e = hint[gid >> SH];
    while (R[e + 1].start <= gid) ++e;
    return e;
}
__device__ __forceinline__ int find_box(const RegionBox* __restrict__ R, int ne, long gid) {
    return find_piece<REGION_HINT>(R, ne, gid);
}

// element l of a piece of extents n at lo, x fastest
__device__ __forceinline__ void piece_ijk(const int* __restrict__ lo, const int* __restrict__ n, const PieceDiv& v,
                                          long l, int& i, int& j, int& k) {
    if (v.sh[0] == -2) {
        const long q = l / n[0], q2 = q / n[1];
        i = lo[0] + (int)(l - q * n[0]);
        j = lo[1] + (int)(q - q2 * n[1]);
        k = lo[2] + (int)q2;
        return;
    }
    const unsigned u = (unsigned)l;
    const unsigned q = v.m[0] ? __umulhi(u, v.m[0]) >> v.sh[0] : u;
    const unsigned q2 = v.m[1] ? __umulhi(q, v.m[1]) >> v.sh[1] : q;
    i = lo[0] + (int)(u - q * (unsigned)n[0]);
    j = lo[1] + (int)(q - q2 * (unsigned)n[1]);
    k = lo[2] + (int)q2;
}
__device__ __forceinline__ void region_ijk(const RegionBox& r, long l, int& i, int& j, int& k) {
    piece_ijk(r.lo, r.n, r.dv, l, i, j, k);
}

// Programmatic dependent launch: a kernel lets the next one of its stream start at once (its
// blocks take the places that drain, find their elements in the constant tables) and itself
// waits here until everything before it is complete and visible.  Nothing but those
// tables may be read before MADV_WAIT, and every kernel that launch_next starts has it.
#define MADV_LET_NEXT() asm volatile("griddepcontrol.launch_dependents;" ::: "memory")
#define MADV_WAIT() asm volatile("griddepcontrol.wait;" ::: "memory")

// Common launch prologue: returns for threads past the range.
// MADV_ELEMENT_OF: the element of block bx (kernels that put components into the block index).
#define MADV_ELEMENT(R, ne, g0, g1, b, i, j, k) MADV_ELEMENT_OF(blockIdx.x, R, ne, g0, g1, b, i, j, k)
#define MADV_ELEMENT_OF(bx, R, ne, g0, g1, b, i, j, k)                     \
    MADV_PIECE(bx, R, ne, g0, g1, b, i, j, k);                            \
    MADV_WAIT()
// (what a kernel needs of its piece is read before the wait: part_ is the piece's pad)
#define MADV_PIECE(bx, R, ne, g0, g1, b, i, j, k)                          \
    MADV_LET_NEXT();                                                      \
    const long gid_ = (g0) + (long)(bx) * blockDim.x + threadIdx.x;        \
    if (gid_ >= (g1)) return;                                             \
    const int e_ = find_box((R), (ne), gid_);                             \
    const int b = (R)[e_].b;                                              \
    [[maybe_unused]] const int part_ = (R)[e_].pad;                        \
    int i, j, k;                                                          \
    region_ijk((R)[e_], gid_ - (R)[e_].start, i, j, k)

// The cells (i, j, k .. k1 - 1) of a thread of a column region (region_columns); COL = false: of a
// region as it is, one cell
#define MADV_COLUMN(COL, R, ne, g0, g1, b, i, j, k, k1)                    \
    MADV_PIECE(blockIdx.x, R, ne, g0, g1, b, i, j, k);                     \
    const int klo_ = (R)[e_].lo[2];                                       \
    const int len_ = (COL) ? (R)[e_].len : 1;                              \
    const int kend_ = klo_ + ((COL) ? (R)[e_].ext : (R)[e_].n[2]);         \
    if (COL) k = klo_ + (k - klo_) * len_;                                 \
    const int k1 = (COL) ? min(k + len_, kend_) : k + 1;                   \
    MADV_WAIT()

// amrex::min / amrex::max (std::min / std::max semantics).  (An integer-key form measured
// slower: the FP64 min/max instruction is not the costly part of the FP64 pipe.)
__device__ __forceinline__ double mn(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double mx(double a, double b) { return (a < b) ? b : a; }

}  // namespace madv
