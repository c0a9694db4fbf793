// madv_ppm_noalloc: Maestro::PPM on one box without a context and without allocating any
// device memory.
//
// Who needs it.  Some callers cannot call cudaMalloc at the point where they run PPM:
// an AMReX application usually reserves most of the GPU's memory for its own arena at
// start-up, so a third-party cudaMalloc there fails or eats into what is left; and code
// that must stay asynchronous cannot afford the implicit device synchronisation that
// cudaMalloc / cudaFree perform.  The single-box PPM keeps its intermediates in registers and
// shared memory, so this entry point holds no memory of its own and calls on different
// streams do not meet.
//
// The size limit is kept for its callers' sake alone: it was that of a static array of
// MADV_PPM_NOALLOC_MAX_DOUBLES doubles of intermediates, which is gone.  A box up to 66 x 66 x 66
// cells (a 64^3 box grown by one cell, the box the reference passes to PPM) is accepted, a
// larger one is rejected with MADV_ERR_LAYOUT before anything runs, as before.
#include "madv_ctx.hpp"

using namespace madv;

// The limit's measure: doubles of one direction's interface values (n_d + 4 faces), van Leer slopes
// (n_d + 2 cells) and two tracing coefficients (n_d + 1 faces), the worst of the three.
static long intermediates(const int n[3]) {
    long worst = 0;
    for (int d = 0; d < 3; ++d) {
        long t = 1;
        for (int e = 0; e < 3; ++e)
            if (e != d) t *= n[e];
        const long need = t * ((n[d] + 4) + (n[d] + 2) + 2 * (n[d] + 1));
        worst = need > worst ? need : worst;
    }
    return worst;
}

extern "C" int madv_ppm_noalloc(const madv_params* params, const madv_box* bx, const madv_fab* s, int comp,
                                const madv_fab* u, const madv_fab* v, const madv_fab* w, int is_umac, const int* bc,
                                const madv_fab* Ip, const madv_fab* Im, void* stream) {
    if (!params || !bx) return MADV_ERR_PARAM;
    if (!(params->dt > 0.0) || !(params->rel_eps >= 0.0) || !(params->dx[0] > 0.0) || !(params->dx[1] > 0.0) ||
        !(params->dx[2] > 0.0)) {
        set_error("madv_ppm_noalloc: dt and dx must be > 0, rel_eps >= 0");
        return MADV_ERR_PARAM;
    }
    int n[3];
    for (int d = 0; d < 3; ++d) {
        n[d] = bx->hi[d] - bx->lo[d] + 1;
        if (n[d] <= 0) {
            set_error("madv_ppm_noalloc: empty box");
            return MADV_ERR_LAYOUT;
        }
    }
    const long need = intermediates(n);
    if (need > (long)MADV_PPM_NOALLOC_MAX_DOUBLES) {
        set_error("madv_ppm_noalloc: the box has " + std::to_string(need) + " doubles of intermediates, past the static " +
                  "limit of " + std::to_string((long)MADV_PPM_NOALLOC_MAX_DOUBLES) +
                  " (boxes up to 66 x 66 x 66 cells fit); use madv_ppm for larger boxes");
        return MADV_ERR_LAYOUT;
    }
    long launches = 0;
    return ppm_box_run(*params, bx, s, comp, u, v, w, is_umac, bc, Ip, Im, (cudaStream_t)stream, launches);
}
