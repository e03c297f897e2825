// claw2_acoustics.cu -- the unsplit step of the acoustics solvers: kernels and
// launch (claw2_march.cuh has the body).
#include <cuda_runtime.h>

#include "claw2_launch.cuh"
#include "claw2_march.cuh"

namespace claw2 {

template <class RP, int MINB>
__global__ void __launch_bounds__(MARCH_NT, MINB) march_step_kernel(StepArgs a, int rows)
{
    chain_wait();
    const TileId t{(int)blockIdx.x, (int)blockIdx.y, (int)gridDim.x, (int)gridDim.y,
                   (int)(blockIdx.y * gridDim.x + blockIdx.x), (int)(gridDim.x * gridDim.y)};
    march_tile<RP, true>(a, t, rows);
}

// Rows of a CTA's tile, for `cols` strips of my rows.  A CTA takes rows + 3 iterations, each a chain of
// dependent FP64 operations (about 1.2 us however few CTAs an SM holds, 1.6 us
// with all it can), so the step is shortest when the grid just fills the SMs
// once; a tile of more than `most` rows is split into more waves instead, whose
// CTAs even out as they retire.  Measured per step, rows 1 / 3 / 4 / 8: variable
// coefficients on 256 x 256 25.1 / 17.7 / 19.3 / 26.2 us (860 CTAs at 3 rows fill
// 8 x 148 slots); rows 12 / 16 / 32 / 64 on 1024 x 1024 76.0 / 76.6 / 73.1 / 103.6.
int march_rows_per_cta(int rp, long long cols, int my)
{
    const bool vc = rp == CLAW2_RP_VC_ACOUSTICS;
    const long long slots = 148LL * (vc ? MarchVc::MINB : MarchConst::MINB);
    const int most = vc ? 32 : 24;
    long long rows = most;
    for (long long waves = 1; waves <= 16; waves++) {
        const long long per_col = waves * slots / cols;             // CTAs a strip may have
        const long long r = per_col > 0 ? (my + per_col - 1) / per_col : most + 1;
        if (r <= most) { rows = r; break; }
    }
    if ((my + rows - 1) / rows > 65535) rows = (my + 65534) / 65535;        // the grid's second dimension
    return (int)rows;
}

int launch_march(int rp, const StepArgs& a0, cudaStream_t st, bool chained)
{
    StepArgs a = a0;
    // the CFL cell: eight of the header's bytes behind the arrival counter
    a.partials = reinterpret_cast<double*>(a.ticket) + 1;
    const int cols = (a.mx + MARCH_TX - 1) / MARCH_TX, rows = march_rows_per_cta(rp, cols, a.my);
    const dim3 grid(cols, (a.my + rows - 1) / rows);
    if (rp == CLAW2_RP_VC_ACOUSTICS)
        return launch_kernel(march_step_kernel<RpVcAcoustics, MarchVc::MINB>, grid, MARCH_NT, 0, st, chained, a, rows);
    return launch_kernel(march_step_kernel<RpAcoustics, MarchConst::MINB>, grid, MARCH_NT, 0, st, chained, a, rows);
}

}  // namespace claw2
