// claw2_lean.cu -- the step of the Euler and shallow-water solvers: kernels and
// launch (claw2_lean.cuh has the body).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "../../include/claw2.h"
#include "claw2_devattr.h"
#include "claw2_launch.cuh"
#include "claw2_lean.cuh"

namespace claw2 {

// tm0 / tm1: tensor maps of the input state (see lean_tiles), passed as
// __grid_constant__ parameters so the TMA unit can read them in place.
// LISTED: as many CTAs as the chip holds step the tiles that lean_scan_kernel listed.
// LOOK: one-state tiles are looked for here.
template <class RP, int T, int NT, bool SPLIT, bool LISTED, bool LOOK>
__global__ void __launch_bounds__(NT, 512 / NT)
lean_step_kernel(StepArgs a, const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1)
{
    extern __shared__ double smem_dyn[];
    __shared__ __align__(8) uint64_t halo_bar;
    chain_wait();
    DevCtx ctx{smem_dyn};
    lean_tiles<RP, T, NT, SPLIT, LOOK, LISTED>(a, ctx, &tm0, &tm1, &halo_bar);
}

// The tiles of a large grid, a warp each: one-state tiles are done, the others listed.
constexpr int SCAN_NT = 256;

template <class RP, int T>
__global__ void __launch_bounds__(SCAN_NT, 4) lean_scan_kernel(StepArgs a, int ntiles)
{
    __shared__ double red[SCAN_NT / 32];
    chain_wait();
    const double* qin = a.qin;
    double* qout = a.qout;
    double dt = a.dt;
    if (a.ctrl) {
        const int done = a.ctrl->done, cur = a.ctrl->cur;           // loaded together
        dt = a.ctrl->dt;
        if (done) return;                          // uniform across the grid
        qin = cur ? a.q1 : a.q0;
        qout = cur ? a.q0 : a.q1;
    }
    const int tile = blockIdx.x * (SCAN_NT / 32) + threadIdx.x / 32;
    double c = 0.0;
    if (tile < ntiles) c = lean_scan_tile<RP, T>(a, qin, qout, tile, dt / a.dx, dt / a.dy);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x / 32] = c;
    __syncthreads();
    if (threadIdx.x != 0) return;
#pragma unroll
    for (int w = 1; w < SCAN_NT / 32; w++) c = c > red[w] ? c : red[w];
    // CFL numbers are >= 0: their bits order as integers (collect_cfl)
    if (c > 0.0) atomicMax(reinterpret_cast<unsigned long long*>(a.partials), (unsigned long long)__double_as_longlong(c));
}

namespace {

// cuTensorMapEncodeTiled from the driver, found through the runtime (no link
// against libcuda, so the library still loads on a machine without a GPU)
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
    static std::atomic<void*> fn{nullptr};
    void* f = fn.load(std::memory_order_acquire);
    if (!f) {
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !f)
            return nullptr;
        fn.store(f, std::memory_order_release);
    }
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
}

// Tensor map of one state buffer for the lean body's halo boxes: the ghosted
// planes (mx+4 columns, my+4 rows, meqn fields; rows ld doubles apart, planes
// `plane` doubles apart), boxes of 16 x rows x meqn, 128-byte swizzle, zeros
// outside the ghosted array.
int halo_tensor_map(CUtensorMap* m, const double* q, const StepArgs& a, int meqn, int rows)
{
    auto encode = tensor_map_encoder();
    if (!encode) return CLAW2_ERR_CUDA;
    if ((reinterpret_cast<uintptr_t>(q) & 15u) != 0) return CLAW2_ERR_INVALID;
    const cuuint64_t dims[3] = {(cuuint64_t)(a.mx + 2 * CLAW2_NUM_GHOST), (cuuint64_t)(a.my + 2 * CLAW2_NUM_GHOST),
                                (cuuint64_t)meqn};
    const cuuint64_t strides[2] = {(cuuint64_t)a.ld * sizeof(double), (cuuint64_t)a.plane * sizeof(double)};
    const cuuint32_t box[3] = {16, (cuuint32_t)rows, (cuuint32_t)meqn};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double*>(q), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? CLAW2_OK : CLAW2_ERR_CUDA;
}

// chained: the previous operation in the stream is a step kernel of the same
// device loop (launch_kernel).
template <class RP, int T, int NT, bool SPLIT, bool LISTED, bool LOOK>
int launch_lean_t(const StepArgs& a, cudaStream_t st, bool chained)
{
    using SM = LeanSmem<RP, T, NT, SPLIT>;
    auto kern = lean_step_kernel<RP, T, NT, SPLIT, LISTED, LOOK>;
    static std::atomic<uint64_t> optin{0};
    if (smem_optin(optin, kern, SM::bytes) != cudaSuccess) return CLAW2_ERR_CUDA;
    CUtensorMap tm0, tm1;
    int rc = halo_tensor_map(&tm0, a.ctrl ? a.q0 : a.qin, a, RP::MEQN, SM::TR);
    if (!rc) rc = a.ctrl ? halo_tensor_map(&tm1, a.q1, a, RP::MEQN, SM::TR) : (tm1 = tm0, CLAW2_OK);
    if (rc) return rc;
    const int n = ((a.mx + T - 1) / T) * ((a.my + T - 1) / T);
    if constexpr (LISTED) {
        constexpr int per = SCAN_NT / 32, most = 148 * (512 / NT);
        rc = launch_kernel(lean_scan_kernel<RP, T>, dim3((n + per - 1) / per), SCAN_NT, 0, st, chained, a, n);
        if (rc) return rc;
        return launch_kernel(kern, dim3(n < most ? n : most), NT, SM::bytes, st, chained, a, tm0, tm1);
    } else {
        return launch_kernel(kern, dim3(n), NT, SM::bytes, st, chained, a, tm0, tm1);
    }
}

// Tiles, block size and pass over one-state tiles.  A chunk of 16 warps takes about
// 7 us unsplit (6 split) and a tile of 28 x 28 cells four of them, whatever the grid;
// one of 12 x 12 (two lines a warp, 8 warps) takes two, shorter with fewer warps on the
// SM, but computes 1.27 times the lines per cell.
//  - 12 x 12 up to 3 tiles per SM of a B200, where most SMs would idle or hold
//    one large tile.  us a step, 12 / 28, Euler 4-wave: 64 x 48 15.3 / 30.4 (24
//    small tiles), 320 x 80 17.9 / 29.9 (189), 320 x 160 22.7 / 29.7 (378), and
//    beyond the line 641 x 163 35.1 / 30.4 (756); split 12.3 / 23.3, 14.3 / 22.7,
//    19.6 / 23.7, and 27.4 / 23.3; shallow water 320 x 160 20.7 / 21.1.
//  - 28 x 28 with 512 threads, one CTA per SM, up to one tile per SM, and for Euler up
//    to 8: the lowest latency of a wave (641 x 163, 138 tiles, 30.4 us against 50.6
//    with 256; the developed shock bubble of 1280 x 320, 552 tiles of uneven cost, 126
//    / 153; shallow water 500 x 333, 216 tiles, 39.6 / 37.2).  In one wave the slowest
//    tile decides, so nobody looks for one-state tiles (256 x 256 28.4 against 29.9,
//    5-wave 32.5 against 35.2).
//  - 28 x 28 with 256 threads, two CTAs per SM, beyond: one CTA's waits (its halo
//    copy, its barriers, the launch of the next CTA) overlap the other's work.
//    512 / 256 on 1500^2 300.9 / 280.4, split 219 / 175, shallow water 328 / 285.  Not
//    the unsplit 5-wave solver: its spilled registers miss the L1 that two CTAs'
//    shared memory leaves (373 / 406).
//  - from 16 tiles per SM on, a pass of its own (lean_scan_kernel) steps the one-state
//    tiles and lists the others, whose kernel then holds fewer registers.  Shallow
//    water 4096^2 at rest around a dam 461 -> 230; no tile at rest, 1500^2: Euler
//    290 -> 262 and 376 -> 314, shallow water 296 -> 297, split 182 -> 190, 220 -> 222
//    and 187 -> 190.  At 1280 x 900 (1518 tiles) shallow water still loses 156 -> 170.
constexpr int SMALL_T = 12;
constexpr long long SMALL_TILES = 3 * 148, LIST_TILES = 16 * 148;

template <class RP, bool SPLIT>
int launch_lean_rp(const StepArgs& a, cudaStream_t st, bool chained)
{
    auto count = [&](int t) { return (long long)((a.mx + t - 1) / t) * ((a.my + t - 1) / t); };
    constexpr bool euler = RP::MEQN > 3, small_l1 = RP::MEQN == 5 && !SPLIT;
    const long long n = count(LEAN_T);
    if (count(SMALL_T) <= SMALL_TILES) return launch_lean_t<RP, SMALL_T, 256, SPLIT, false, true>(a, st, chained);
    if (n <= 148) return launch_lean_t<RP, LEAN_T, 512, SPLIT, false, false>(a, st, chained);
    if (n > LIST_TILES && !a.src) return launch_lean_t<RP, LEAN_T, euler && !SPLIT ? 512 : 256, SPLIT, true, false>(a, st, chained);
    if constexpr (euler)
        if (small_l1 || n <= 8 * 148) return launch_lean_t<RP, LEAN_T, 512, SPLIT, false, true>(a, st, chained);
    if constexpr (!small_l1) return launch_lean_t<RP, LEAN_T, 256, SPLIT, false, true>(a, st, chained);
    return CLAW2_ERR_INVALID;                      // not reached
}

template <class RP>
int launch_lean_form(const StepArgs& a, bool split, cudaStream_t st, bool chained)
{
    return split ? launch_lean_rp<RP, true>(a, st, chained) : launch_lean_rp<RP, false>(a, st, chained);
}

}  // namespace

int launch_lean(int rp, bool split, const StepArgs& a0, cudaStream_t st, bool chained)
{
    StepArgs a = a0;
    // the CFL cell: eight of the header's bytes behind the arrival counter
    a.partials = reinterpret_cast<double*>(a.ticket) + 1;
    a.list = reinterpret_cast<int*>(a.ticket + 16);        // behind the header: as many ints as it has 28-tiles fit
    switch (rp) {
    case CLAW2_RP_EULER_4WAVE: return launch_lean_form<RpEuler<false>>(a, split, st, chained);
    case CLAW2_RP_EULER_5WAVE: return launch_lean_form<RpEuler<true>>(a, split, st, chained);
    case CLAW2_RP_SHALLOW_ROE: return launch_lean_form<RpShallow>(a, split, st, chained);
    default: return CLAW2_ERR_INVALID;
    }
}

}  // namespace claw2
