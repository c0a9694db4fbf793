// Launch helper shared by the kernel files: one launch over the region pieces of every box
// (batched), or one launch per piece (the per-box form of the reference's MFIter loop).
#pragma once
#include "madv_ctx.hpp"

namespace madv {

#define KARGS const RegionBox *__restrict__ R, int ne, long g0, long g1, const FabView *__restrict__ V, int nb
#define VW(f) V[(f) * nb + b]

static constexpr int TPB = 256;

// Starts a kernel that opens with MADV_LET_NEXT / MADV_WAIT.  On a stream it is a programmatic
// dependent of the kernel before it: a chain of small kernels goes from 4.1 to 1.5 us a
// kernel.  In a graph the nodes follow each other in 1.1 us either way, and past 10^6
// elements the early start costs (4.7 against 3.5 us a kernel), so captured launches are
// plain.
template <typename... P, typename... Args>
static inline void launch_on(cudaStream_t st, bool plain, dim3 grid, int tpb, void (*kern)(P...), Args... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)tpb);
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = plain ? 0 : 1;
    cudaLaunchKernelEx(&cfg, kern, (P)args...);
}
template <typename... P, typename... Args>
static inline void launch_next(const Ctx& c, dim3 grid, int tpb, void (*kern)(P...), Args... args) {
    launch_on(c.stream, c.capturing, grid, tpb, kern, args...);
}

// One launch over every box (batched), or one launch per region piece (per-box mode, the
// MFIter + ParallelFor form of the reference).  Kernel arguments after the region are
// (V, nb, ...).  Threads per block: the kernel's autotuned value on this level.
// per_warp > 0: kernels whose warps advance by that many elements instead of 32.
// gq components are interleaved in the block index, so that the blocks of one place run together
// and share what they read.
template <typename Kern, typename... Args>
static inline void launch(Ctx& c, const RegionTable& rt, int gq, Kern kern, int per_warp, const FabView* V, Args... args) {
    const int tpb = c.tpb_of((const void*)kern);  // before a dry return: no attribute query while capturing
    if (rt.total == 0 || c.dry) return;
    const int ne = (int)rt.h.size();
    auto grid = [&](long n) {
        const long threads = per_warp ? (n + per_warp - 1) / per_warp * 32 : n;
        return dim3((unsigned)((threads + tpb - 1) / tpb * gq));
    };
    if (!c.per_box) {
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        if (c.profiling) {
            e0 = c.next_event();
            e1 = c.next_event();
            cudaEventRecord(e0, c.stream);
        }
        launch_next(c, grid(rt.total), tpb, kern, (const RegionBox*)rt.d, ne, 0L, rt.total, V, c.nb, args...);
        if (c.profiling) {
            cudaEventRecord(e1, c.stream);
            c.prof.push_back({(const void*)kern, e0, e1});
        }
        c.launches++;
    } else {
        for (int e = 0; e < ne; ++e) {
            long s0 = rt.h[e].start;
            long s1 = (e + 1 < ne) ? rt.h[e + 1].start : rt.total;
            if (s1 <= s0) continue;
            launch_next(c, grid(s1 - s0), tpb, kern, (const RegionBox*)rt.d, ne, s0, s1, V, c.nb, args...);
            c.launches++;
        }
    }
}
template <typename Kern, typename... Args>
static inline void launch(Ctx& c, const RegionTable& rt, int gq, Kern kern, const FabView* V, Args... args) {
    launch(c, rt, gq, kern, 0, V, args...);
}

// Region helpers: the valid box grown by g, and face boxes.
static inline const RegionTable& rg_grow(Ctx& c, int g, int nodal = -1) { return region(c, g, g, g, g, g, g, nodal); }

}  // namespace madv
