// claw2_host.h -- host helpers shared by the translation units that launch steps.
#pragma once

#include <cuda_runtime.h>

#include <cstring>

#include "../../include/claw2.h"
#include "claw2_kernels.cuh"

namespace claw2 {

inline cudaStream_t S(void* s) { return reinterpret_cast<cudaStream_t>(s); }

inline int solver_shape(int rp, int* meqn, int* mw, int* maux)
{
    switch (rp) {
    case CLAW2_RP_ACOUSTICS: *meqn = 3; *mw = 2; *maux = 0; return 0;
    case CLAW2_RP_VC_ACOUSTICS: *meqn = 3; *mw = 2; *maux = 2; return 0;
    case CLAW2_RP_EULER_4WAVE: *meqn = 4; *mw = 4; *maux = 0; return 0;
    case CLAW2_RP_EULER_5WAVE: *meqn = 5; *mw = 5; *maux = 0; return 0;
    case CLAW2_RP_SHALLOW_ROE: *meqn = 3; *mw = 3; *maux = 0; return 0;
    case CLAW2_RP_PSYSTEM: *meqn = 3; *mw = 2; *maux = 4; return 0;
    default: return -1;
    }
}

inline bool periodic_ok(int bl, int bu) { return (bl == CLAW2_BC_PERIODIC) == (bu == CLAW2_BC_PERIODIC); }

inline bool fused_ghosts(const claw2_problem* p)
{
    for (int d = 0; d < 2; d++) {
        if (p->bc_lower[d] == CLAW2_BC_CUSTOM || p->bc_upper[d] == CLAW2_BC_CUSTOM) return false;
        if (!periodic_ok(p->bc_lower[d], p->bc_upper[d])) return false;
    }
    return p->mx >= 4 && p->my >= 4;
}

// Custom sides do not keep a tile body from writing the other sides' ghost cells
// (write_custom_corners has the corners beside them).
inline bool fused_beside_custom(const claw2_problem* p)
{
    for (int d = 0; d < 2; d++)
        if (!periodic_ok(p->bc_lower[d], p->bc_upper[d])) return false;
    return p->mx >= 4 && p->my >= 4;
}

inline void fill_args(const claw2_problem* p, double* q, StepArgs& a)
{
    claw2_layout L;
    claw2_get_layout(p, &L);
    std::memset(&a, 0, sizeof a);
    a.ld = L.ld; a.plane = L.plane;
    a.mx = p->mx; a.my = p->my;
    a.dx = p->dx; a.dy = p->dy;
    a.order = p->order; a.trans = p->transverse; a.capa = p->index_capa; a.fwave = p->use_fwave;
    a.limit_any = 0;
    for (int w = 0; w < CLAW2_MAX_WAVES; w++) {
        a.mthlim[w] = w < p->num_waves ? p->mthlim[w] : 0;
        if (w < p->num_waves && p->mthlim[w] > 0) a.limit_any = 1;
    }
    a.limit_first = a.mthlim[0];
    for (int w = 1; w < 4 && w < p->num_waves; w++)
        if (a.mthlim[w] != a.limit_first) a.limit_first = -1;
    for (int k = 0; k < CLAW2_MAX_PARAMS; k++) a.prm[k] = p->params[k];
    a.ghost_fused = fused_ghosts(p) ? 1 : 0;
    for (int d = 0; d < 2; d++) { a.bcl[d] = p->bc_lower[d]; a.bcu[d] = p->bc_upper[d]; }
    (void)q;
}

}  // namespace claw2
