// claw2_acoustics.cu -- the step of the acoustics solvers: kernels and launch
// (claw2_march.cuh has the unsplit body, claw2_rows.cuh the split one).
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "claw2_devattr.h"
#include "claw2_launch.cuh"
#include "claw2_march.cuh"
#include "claw2_rows.cuh"

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

constexpr int ROWS_NT = 256;

template <bool VC, int T>
__global__ void __launch_bounds__(ROWS_NT, 4) rows_step_kernel(StepArgs a)
{
    extern __shared__ double smem_dyn[];
    chain_wait();
    DevCtx ctx{smem_dyn};
    const TileId t{(int)blockIdx.x, (int)blockIdx.y, (int)gridDim.x, (int)gridDim.y,
                   (int)(blockIdx.y * gridDim.x + blockIdx.x), (int)(gridDim.x * gridDim.y)};
    rows_tile<VC, T, ROWS_NT>(a, ctx, t);
}

template <bool VC, int T>
static int launch_rows_t(const StepArgs& a, cudaStream_t st, bool chained)
{
    using SM = RowsSmem<VC, T, ROWS_NT>;
    auto kern = rows_step_kernel<VC, T>;
    static std::atomic<uint64_t> optin{0};
    if (smem_optin(optin, kern, SM::bytes) != cudaSuccess) return CLAW2_ERR_CUDA;
    return launch_kernel(kern, dim3((a.mx + T - 1) / T, (a.my + T - 1) / T), ROWS_NT, SM::bytes, st, chained, a);
}

// Tiles: a tile of 28 x 28 cells takes eight passes of the CTA's 8 warps over
// lines, one of 12 x 12 (two lines a warp) two, but sweeps 1.37 times the lines per
// cell.  The small ones serve up to 8 of them per SM of a B200, two waves of the 4
// CTAs that an SM holds.  us a step, 12 / 28: acoustics 64 x 48 7.8 / 12.4,
// 256 x 256 10.3 / 15.5, 500 x 300 (1050 small tiles) 13.4 / 16.5, and beyond the
// line 800 x 400 (2278) 23.0 / 21.2, 1500^2 123 / 69; variable coefficients
// 8.1 / 12.8, 10.6 / 16.6, 14.2 / 18.2, 24.5 / 23.0, 132 / 78.
constexpr long long ROWS_SMALL_TILES = 8 * 148;

template <bool VC>
static int launch_rows_c(const StepArgs& a, cudaStream_t st, bool chained)
{
    const long long small = (long long)((a.mx + 11) / 12) * ((a.my + 11) / 12);
    return small <= ROWS_SMALL_TILES ? launch_rows_t<VC, 12>(a, st, chained) : launch_rows_t<VC, 28>(a, st, chained);
}

int launch_rows(int rp, const StepArgs& a0, cudaStream_t st, bool chained)
{
    StepArgs a = a0;
    a.partials = reinterpret_cast<double*>(a.ticket) + 1;           // the CFL cell, as above
    return rp == CLAW2_RP_VC_ACOUSTICS ? launch_rows_c<true>(a, st, chained) : launch_rows_c<false>(a, st, chained);
}

}  // namespace claw2
