// claw2_psystem.cu -- the unsplit step of the p-system: kernels and launch
// (claw2_psystem.cuh has the body).
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "../../include/claw2.h"
#include "claw2_devattr.h"
#include "claw2_launch.cuh"
#include "claw2_psystem.cuh"

namespace claw2 {

// TALL: more rows of tiles than a grid's second dimension holds, in one dimension.
template <int T, int NT, bool TALL>
__global__ void __launch_bounds__(NT, 512 / NT) psystem_step_kernel(StepArgs a)
{
    extern __shared__ double smem_dyn[];
    chain_wait();
    DevCtx ctx{smem_dyn};
    TileId t{(int)blockIdx.x, (int)blockIdx.y, (int)gridDim.x, (int)gridDim.y,
             (int)(blockIdx.y * gridDim.x + blockIdx.x), (int)(gridDim.x * gridDim.y)};
    if constexpr (TALL) {
        t.nbx = (a.mx + T - 1) / T;
        t.nby = t.ntiles / t.nbx;
        t.bx = t.part % t.nbx;
        t.by = t.part / t.nbx;
    }
    psys_tile<T, NT>(a, ctx, t);
}

template <int T, int NT, bool TALL = false>
static int launch_psystem_t(const StepArgs& a, cudaStream_t st, bool chained)
{
    auto kern = psystem_step_kernel<T, NT, TALL>;
    static std::atomic<uint64_t> optin{0};
    if (smem_optin(optin, kern, PsysSmem<T, NT>::bytes) != cudaSuccess) return CLAW2_ERR_CUDA;
    const int nbx = (a.mx + T - 1) / T, nby = (a.my + T - 1) / T;
    return launch_kernel(kern, TALL ? dim3(nbx * nby) : dim3(nbx, nby), NT, PsysSmem<T, NT>::bytes, st, chained, a);
}

// Tiles and block size, as in claw2_lean.cu.  us a step, 12 x 12 / 28 x 28 with 512
// threads / with 256: 64 x 48 11.3 / 18.2 / 25.3, 200 x 200 (289 small tiles) 12.0 /
// 18.3 / 26.3, 256 x 256 (484) 16.0 / 18.1 / 25.6, and beyond the first line
// 641 x 163 (756 small, 138 large) 21.1 / 17.2 / 26.3, 800 x 400 (435 large) 48.2 /
// 36.4 / 40.0, beyond the second 600 x 600 (484) 55.8 / 45.4 / 44.0, 1500^2 307 /
// 211 / 182.
constexpr long long PSYS_SMALL_TILES = 4 * 148, PSYS_BIG_BLOCK_TILES = 3 * 148;

int launch_psystem(const StepArgs& a0, cudaStream_t st, bool chained)
{
    StepArgs a = a0;
    // the CFL cell: eight of the header's bytes behind the arrival counter
    a.partials = reinterpret_cast<double*>(a.ticket) + 1;
    auto count = [&](int t) { return (long long)((a.mx + t - 1) / t) * ((a.my + t - 1) / t); };
    if (count(12) <= PSYS_SMALL_TILES) return launch_psystem_t<12, 256>(a, st, chained);
    if (count(28) <= PSYS_BIG_BLOCK_TILES) return launch_psystem_t<28, 512>(a, st, chained);
    // 65535 rows of tiles (one dimension for all makes 200 x 200 2% slower)
    if (a.my > 65535 * 28) return launch_psystem_t<28, 256, true>(a, st, chained);
    return launch_psystem_t<28, 256>(a, st, chained);
}

}  // namespace claw2
