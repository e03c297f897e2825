// claw2_batch.cu -- the batched form: many independent instances per launch.
//
// Built like claw2_capi.cu (sm_100a, no FMA contraction).
#include <cuda_runtime.h>

#include <atomic>

#define CLAW2_EXPORT __attribute__((visibility("default")))
#include "../../include/claw2.h"
#include "claw2_devattr.h"
#include "claw2_host.h"
#include "claw2_kernels.cuh"
#include "claw2_launch.cuh"
#include "claw2_light.cuh"
#include "claw2_march.cuh"

namespace claw2 {

// The two-wave acoustics solvers have leaner bodies of the unsplit step: a tile
// body (claw2_light.cuh) and a marching one (claw2_march.cuh).
template <class RP> struct HasLight { static constexpr bool value = false; };
template <> struct HasLight<RpAcoustics> { static constexpr bool value = true; };
template <> struct HasLight<RpVcAcoustics> { static constexpr bool value = true; };

// Instance of tile t: the last one with tile_begin <= t (binary search).
// With tb (the instances' tile_begin copied into shared memory by the
// kernel) the search reads shared memory instead of walking the descriptors
// in global memory, a chain of dependent L2 loads per tile.
__device__ __forceinline__ int batch_instance_of(const claw2_batch_instance* __restrict__ inst, int ninst, int t,
                                                 const int* tb = nullptr)
{
    int lo = 0, hi = ninst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((tb ? tb[mid] : __ldg(&inst[mid].tile_begin)) <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Instance of tile t from the caller's map (one load); without a map, or where
// its entry does not hold tile t, by search.
__device__ __forceinline__ int batch_instance_of_tile(const claw2_batch_instance* __restrict__ inst, int ninst, int t,
                                                      const int32_t* __restrict__ tile_inst)
{
    const int k = tile_inst ? __ldg(&tile_inst[t]) : -1;
    if (k < 0 || k >= ninst || t < inst[k].tile_begin || t - inst[k].tile_begin >= inst[k].nbx * inst[k].nby)
        return batch_instance_of(inst, ninst, t);
    return k;
}

// batches of at most this many instances keep their tile_begin table in
// shared memory (4 bytes each)
constexpr int kBatchTableMax = 4096;

// Instance of tile t + 1 given k, the instance of tile t: tile_begin is
// non-decreasing, so it is the last instance at or after k whose tile_begin is
// <= t + 1 (the same one or, crossing an instance's last tile, the next one
// with tiles).
__device__ __forceinline__ int batch_instance_after(const claw2_batch_instance* __restrict__ inst, int ninst, int k,
                                                    int t, const int* tb)
{
    while (k + 1 < ninst && (tb ? tb[k + 1] : __ldg(&inst[k + 1].tile_begin)) <= t + 1) k++;
    return k;
}

// Ask L2 for the input halo of tile t (instance k; rows j0-2..j0+TY+1 and
// columns i0-2..i0+TX+1, clipped to the ghosted arrays, of the current state
// and of aux) while the CTA works on the tile before it: an instance's data is
// read once per step, from HBM, so the tile's first loads would otherwise wait
// for DRAM.  One prefetch per 128-byte line, spread over the CTA's threads.
// The addresses stay inside the instance's arrays; results do not depend on
// it.
template <int MEQN, int MAUX, int TX, int TY, int NT>
__device__ __forceinline__ void batch_prefetch_tile(const claw2_batch_instance* __restrict__ inst, int k, int t)
{
    const claw2_batch_instance& I = inst[k];
    const claw2_control* c = I.ctrl;
    if (c->done) return;
    const double* q = c->cur ? I.q1 : I.q0;
    const int lt = t - I.tile_begin;
    const int i0 = (lt % I.nbx) * TX, j0 = (lt / I.nbx) * TY;
    const int rlo = j0 - 2, rhi = (j0 + TY + 1 < I.my + 1) ? j0 + TY + 1 : I.my + 1;
    const int clo = i0 - 2, chi = (i0 + TX + 1 < I.mx + 1) ? i0 + TX + 1 : I.mx + 1;
    // byte range of one row segment, in whole 128-byte lines
    const long long b0 = (long long)(clo + CLAW2_NUM_GHOST) * 8, b1 = (long long)(chi + CLAW2_NUM_GHOST) * 8 + 8;
    const int l0 = (int)(b0 >> 7), nl = (int)((b1 + 127) >> 7) - l0;
    const int nrow = rhi - rlo + 1;
    // one (field, row) per thread, its 128-byte lines in turn
    for (int rf = threadIdx.x; rf < (MEQN + MAUX) * nrow; rf += NT) {
        const int r = rf % nrow, f = rf / nrow;
        const char* base = f < MEQN ? (const char*)(q + f * I.plane) : (const char*)(I.aux + (f - MEQN) * I.plane);
        const char* row = base + (long long)(rlo + r + CLAW2_NUM_GHOST) * I.ld * 8 + ((long long)l0 << 7);
        for (int line = 0; line < nl; line++) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + (line << 7)));
    }
}

// Batched step: a persistent grid walks the concatenated tile list of all
// instances; each tile (T x T cells) is one tile-body call with that
// instance's buffers, with an L2 prefetch of the CTA's next tile issued first.
// body_doubles: the tile body's shared memory; with `table` set the
// instances' tile_begin table follows it.
template <class RP, int NT, int MINB, bool LIGHT, int T>
__global__ void __launch_bounds__(NT, MINB)
batch_kernel(const claw2_batch_instance* __restrict__ inst, int ninst, int ntiles, StepArgs common, int body_doubles,
             int table)
{
    static_assert(LIGHT || T == 29, "the generic body runs 29x29 tiles in the batch");
    extern __shared__ double smem_dyn[];
    DevCtx ctx{smem_dyn};
    int* tb = nullptr;
    if (table) {
        tb = reinterpret_cast<int*>(smem_dyn + body_doubles);
        for (int i = threadIdx.x; i < ninst; i += NT) tb[i] = __ldg(&inst[i].tile_begin);
        __syncthreads();
    }
    // each CTA takes a contiguous run of tiles: consecutive tiles mostly
    // belong to the same instance (its descriptor and controller stay in L1)
    // and share halo lines with the tile before them
    const int tbeg = (int)((long long)ntiles * blockIdx.x / gridDim.x);
    const int tend = (int)((long long)ntiles * (blockIdx.x + 1) / gridDim.x);
    // the run's first instance by binary search, then one step at a time
    int lo = tbeg < tend ? batch_instance_of(inst, ninst, tbeg, tb) : 0;
    for (int t = tbeg; t < tend; t++) {
        const int nxt = t + 1 < tend ? batch_instance_after(inst, ninst, lo, t, tb) : lo;
        if (t + 1 < tend) batch_prefetch_tile<RP::MEQN, RP::MAUX, T, T, NT>(inst, nxt, t + 1);
        const claw2_batch_instance& I = inst[lo];
        StepArgs a = common;
        a.q0 = I.q0; a.q1 = I.q1; a.aux = I.aux; a.ctrl = I.ctrl;
        a.partials = I.partials; a.ticket = I.ticket;
        a.ld = I.ld; a.plane = I.plane; a.mx = I.mx; a.my = I.my; a.dx = I.dx; a.dy = I.dy;
        a.ghost_fused = (I.mx >= 4 && I.my >= 4) ? common.ghost_fused : 0;
        const int lt = t - I.tile_begin;
        const TileId tile{lt % I.nbx, lt / I.nbx, I.nbx, I.nby, lt, I.nbx * I.nby};
        if constexpr (LIGHT) light_tile_at<RP, T, T, NT>(a, ctx, tile);
        else step_tile_at<RP, 29, 29, NT, false>(a, ctx, tile);
        __syncthreads();                            // shared memory is reused by the next tile
        lo = nxt;
    }
}

// Batched step with one CTA per tile (grid = all tiles of all instances):
// the hardware hands tiles to SMs as slots free up, so uneven tiles balance
// themselves, and no loop state stays live across the tile body.  The tile's
// instance comes from the caller's tile -> instance map when there is one,
// else from a binary search over the descriptors (a chain of dependent L2
// loads at the CTA's start); there is no L2 prefetch of a next tile, the
// other resident CTAs cover the first loads.
template <class RP, int NT, int MINB, bool LIGHT, int T>
__global__ void __launch_bounds__(NT, MINB)
batch_tile_kernel(const claw2_batch_instance* __restrict__ inst, int ninst, StepArgs common,
                  const int32_t* __restrict__ tile_inst)
{
    static_assert(LIGHT || T == 29, "the generic body runs 29x29 tiles in the batch");
    extern __shared__ double smem_dyn[];
    DevCtx ctx{smem_dyn};
    const int t = (int)blockIdx.x;
    const claw2_batch_instance& I = inst[batch_instance_of_tile(inst, ninst, t, tile_inst)];
    StepArgs a = common;
    a.q0 = I.q0; a.q1 = I.q1; a.aux = I.aux; a.ctrl = I.ctrl;
    a.partials = I.partials; a.ticket = I.ticket;
    a.ld = I.ld; a.plane = I.plane; a.mx = I.mx; a.my = I.my; a.dx = I.dx; a.dy = I.dy;
    a.ghost_fused = (I.mx >= 4 && I.my >= 4) ? common.ghost_fused : 0;
    const int lt = t - I.tile_begin;
    const TileId tile{lt % I.nbx, lt / I.nbx, I.nbx, I.nby, lt, I.nbx * I.nby};
    if constexpr (LIGHT) light_tile_at<RP, T, T, NT>(a, ctx, tile);
    else step_tile_at<RP, 29, 29, NT, false>(a, ctx, tile);
}

// The same with the marching body (claw2_march.cuh): tiles of 28 columns by
// `rows` rows, two warps each.
template <class RP, int MINB>
__global__ void __launch_bounds__(MARCH_NT, MINB)
batch_march_kernel(const claw2_batch_instance* __restrict__ inst, int ninst, StepArgs common,
                   const int32_t* __restrict__ tile_inst, int rows)
{
    const int t = (int)blockIdx.x;
    const claw2_batch_instance& I = inst[batch_instance_of_tile(inst, ninst, t, tile_inst)];
    StepArgs a = common;
    a.q0 = I.q0; a.q1 = I.q1; a.aux = I.aux; a.ctrl = I.ctrl;
    a.partials = I.partials; a.ticket = I.ticket;
    a.ld = I.ld; a.plane = I.plane; a.mx = I.mx; a.my = I.my; a.dx = I.dx; a.dy = I.dy;
    a.ghost_fused = (I.mx >= 4 && I.my >= 4) ? common.ghost_fused : 0;
    const int lt = t - I.tile_begin;
    const TileId tile{lt % I.nbx, lt / I.nbx, I.nbx, I.nby, lt, I.nbx * I.nby};
    march_tile<RP, false>(a, tile, rows);
}

}  // namespace claw2

using namespace claw2;

namespace {
// threads per CTA, resident CTAs per SM, tile edge (cells per CTA per work
// item = tile^2).  Variants 4.. exist for the light acoustics body only
// (claw2_batch_advance returns CLAW2_ERR_UNSUPPORTED for them with the other
// solvers); a line of the light body has 32 lanes for tile + 3 interfaces, so
// smaller tiles leave lanes idle but waste fewer cells at instance edges.
// persistent: a grid of SMs x resident CTAs walking contiguous runs of tiles
// (batch_kernel); otherwise one CTA per tile (batch_tile_kernel).  Tile edges
// 28, 14 and 7 are the rows of a tile of the marching body, 28 columns wide.
struct BatchVariant { int threads, minb, tile, persistent; };
constexpr BatchVariant kBatchVariants[] = {{256, 2, 29, 1}, {128, 4, 29, 1}, {128, 3, 29, 1}, {512, 1, 29, 1},
                                           {256, 3, 29, 1}, {256, 4, 29, 1}, {256, 3, 21, 1}, {256, 4, 21, 1},
                                           {256, 3, 13, 1}, {256, 4, 13, 1}, {256, 3, 29, 0}, {256, 4, 29, 0},
                                           {128, 6, 29, 0}, {512, 2, 29, 0}, {64, 8, 28, 0}, {64, 8, 14, 0},
                                           {64, 8, 7, 0}};
constexpr int kNumBatchVariants = sizeof(kBatchVariants) / sizeof(kBatchVariants[0]);

bool batch_march_tile(int tile) { return tile == 28 || tile == 14 || tile == 7; }
bool batch_tile_ok(int tile) { return tile == 29 || tile == 21 || tile == 13 || batch_march_tile(tile); }

template <class RP, int NT, int MINB, bool LIGHT, int T>
int batch_launch_t(const StepArgs& common, const claw2_batch_instance* inst, int ninst, int ntiles, int nsteps,
                   cudaStream_t st)
{
    constexpr int SMB = LIGHT ? LightSmem<T, T, NT>::bytes : TileSmem<RP, 29, 29, NT, false>::bytes;
    constexpr int kSmemLimit = 227 * 1024;        // dynamic shared memory a CTA can opt in to
    constexpr int SMMAX = SMB + 4 * kBatchTableMax < kSmemLimit ? SMB + 4 * kBatchTableMax : SMB;
    auto kern = batch_kernel<RP, NT, MINB, LIGHT, T>;
    static std::atomic<uint64_t> optin{0};
    if (smem_optin(optin, kern, SMMAX) != cudaSuccess) return CLAW2_ERR_CUDA;
    // the persistent grid: SMs x the CTAs that fit with this launch's table
    const int tbytes = (4 * ninst + 15) / 16 * 16;
    const int table = ninst <= kBatchTableMax && SMB + tbytes <= SMMAX;
    const int smem = SMB + (table ? tbytes : 0);
    int dev = 0, nsm = 0, occ = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, NT, smem) != cudaSuccess || occ < 1)
        return CLAW2_ERR_CUDA;
    const int grid = nsm * occ;
    const int g = ntiles < grid ? ntiles : grid;
    for (int n = 0; n < nsteps; n++) {
        kern<<<g, NT, smem, st>>>(inst, ninst, ntiles, common, SMB / 8, table);
        if (cudaGetLastError() != cudaSuccess) return CLAW2_ERR_CUDA;
    }
    return CLAW2_OK;
}

template <class RP, int NT, int MINB, bool LIGHT, int T>
int batch_launch_tiles(const StepArgs& common, const claw2_batch_instance* inst, int ninst, int ntiles, int nsteps,
                       const int32_t* tile_inst, cudaStream_t st)
{
    constexpr int SMB = LIGHT ? LightSmem<T, T, NT>::bytes : TileSmem<RP, 29, 29, NT, false>::bytes;
    auto kern = batch_tile_kernel<RP, NT, MINB, LIGHT, T>;
    static std::atomic<uint64_t> optin{0};
    if (smem_optin(optin, kern, SMB) != cudaSuccess) return CLAW2_ERR_CUDA;
    for (int n = 0; n < nsteps; n++) {
        kern<<<ntiles, NT, SMB, st>>>(inst, ninst, common, tile_inst);
        if (cudaGetLastError() != cudaSuccess) return CLAW2_ERR_CUDA;
    }
    return CLAW2_OK;
}

template <class RP>
int batch_launch_march(const StepArgs& common, const claw2_batch_instance* inst, int ninst, int ntiles, int nsteps,
                       const int32_t* tile_inst, int rows, cudaStream_t st)
{
    for (int n = 0; n < nsteps; n++) {
        batch_march_kernel<RP, MarchOf<RP>::type::MINB><<<ntiles, MARCH_NT, 0, st>>>(inst, ninst, common, tile_inst, rows);
        if (cudaGetLastError() != cudaSuccess) return CLAW2_ERR_CUDA;
    }
    return CLAW2_OK;
}

template <class RP>
int batch_launch_rp(int variant, const StepArgs& c, const claw2_batch_instance* inst, int ninst, int ntiles,
                    int nsteps, const int32_t* tile_inst, cudaStream_t st)
{
    if constexpr (HasLight<RP>::value) {
        if (c.capa < 0 && !c.fwave) {
            switch (variant) {
            case 0: return batch_launch_t<RP, 256, 2, true, 29>(c, inst, ninst, ntiles, nsteps, st);
            case 1: return batch_launch_t<RP, 128, 4, true, 29>(c, inst, ninst, ntiles, nsteps, st);
            case 2: return batch_launch_t<RP, 128, 3, true, 29>(c, inst, ninst, ntiles, nsteps, st);
            case 3: return batch_launch_t<RP, 512, 1, true, 29>(c, inst, ninst, ntiles, nsteps, st);
            case 4: return batch_launch_t<RP, 256, 3, true, 29>(c, inst, ninst, ntiles, nsteps, st);
            case 5: return batch_launch_t<RP, 256, 4, true, 29>(c, inst, ninst, ntiles, nsteps, st);
            case 6: return batch_launch_t<RP, 256, 3, true, 21>(c, inst, ninst, ntiles, nsteps, st);
            case 7: return batch_launch_t<RP, 256, 4, true, 21>(c, inst, ninst, ntiles, nsteps, st);
            case 8: return batch_launch_t<RP, 256, 3, true, 13>(c, inst, ninst, ntiles, nsteps, st);
            case 9: return batch_launch_t<RP, 256, 4, true, 13>(c, inst, ninst, ntiles, nsteps, st);
            case 10: return batch_launch_tiles<RP, 256, 3, true, 29>(c, inst, ninst, ntiles, nsteps, tile_inst, st);
            case 11: return batch_launch_tiles<RP, 256, 4, true, 29>(c, inst, ninst, ntiles, nsteps, tile_inst, st);
            case 12: return batch_launch_tiles<RP, 128, 6, true, 29>(c, inst, ninst, ntiles, nsteps, tile_inst, st);
            case 13: return batch_launch_tiles<RP, 512, 2, true, 29>(c, inst, ninst, ntiles, nsteps, tile_inst, st);
            case 14: case 15: case 16:
                return batch_launch_march<RP>(c, inst, ninst, ntiles, nsteps, tile_inst, kBatchVariants[variant].tile, st);
            default: return CLAW2_ERR_INVALID;
            }
        }
    }
    switch (variant) {
    case 0: return batch_launch_t<RP, 256, 2, false, 29>(c, inst, ninst, ntiles, nsteps, st);
    case 1: return batch_launch_t<RP, 128, 4, false, 29>(c, inst, ninst, ntiles, nsteps, st);
    case 2: return batch_launch_t<RP, 128, 3, false, 29>(c, inst, ninst, ntiles, nsteps, st);
    case 3: return batch_launch_t<RP, 512, 1, false, 29>(c, inst, ninst, ntiles, nsteps, st);
    default: return variant < kNumBatchVariants ? CLAW2_ERR_UNSUPPORTED : CLAW2_ERR_INVALID;
    }
}

int batch_launch(const claw2_problem* p, const claw2_batch_instance* inst, int ninst, int ntiles, int nsteps,
                 int variant, const int32_t* tile_inst, cudaStream_t st)
{
    StepArgs c;
    fill_args(p, nullptr, c);
    c.ghost_fused = 1;
    for (int d = 0; d < 2; d++)
        if (p->bc_lower[d] == CLAW2_BC_CUSTOM || p->bc_upper[d] == CLAW2_BC_CUSTOM) return CLAW2_ERR_UNSUPPORTED;
    switch (p->rp) {
    case CLAW2_RP_ACOUSTICS: return batch_launch_rp<RpAcoustics>(variant, c, inst, ninst, ntiles, nsteps, tile_inst, st);
    case CLAW2_RP_VC_ACOUSTICS: return batch_launch_rp<RpVcAcoustics>(variant, c, inst, ninst, ntiles, nsteps, tile_inst, st);
    case CLAW2_RP_EULER_4WAVE: return batch_launch_rp<RpEuler<false>>(variant, c, inst, ninst, ntiles, nsteps, tile_inst, st);
    case CLAW2_RP_EULER_5WAVE: return batch_launch_rp<RpEuler<true>>(variant, c, inst, ninst, ntiles, nsteps, tile_inst, st);
    case CLAW2_RP_SHALLOW_ROE: return batch_launch_rp<RpShallow>(variant, c, inst, ninst, ntiles, nsteps, tile_inst, st);
    case CLAW2_RP_PSYSTEM: return batch_launch_rp<RpPsystem>(variant, c, inst, ninst, ntiles, nsteps, tile_inst, st);
    default: return CLAW2_ERR_INVALID;
    }
}

int batch_check(const claw2_problem* p, const claw2_batch_instance* inst, int ninst, int ntiles, int nsteps,
                int variant)
{
    if (!p || !inst || ninst < 1 || ntiles < 1 || nsteps < 0) return CLAW2_ERR_INVALID;
    if (variant < 0 || variant >= kNumBatchVariants) return CLAW2_ERR_INVALID;
    if (p->transverse < 0) return CLAW2_ERR_UNSUPPORTED;
    int meqn, mw, maux;
    if (solver_shape(p->rp, &meqn, &mw, &maux) || p->num_eqn != meqn || p->num_waves != mw || p->num_aux < maux)
        return CLAW2_ERR_INVALID;
    if (p->num_ghost != CLAW2_NUM_GHOST || p->index_capa >= p->num_aux) return CLAW2_ERR_INVALID;
    for (int d = 0; d < 2; d++)
        if (!periodic_ok(p->bc_lower[d], p->bc_upper[d])) return CLAW2_ERR_UNSUPPORTED;
    return CLAW2_OK;
}
}  // namespace

extern "C" {

int claw2_batch_num_variants(void) { return kNumBatchVariants; }

int claw2_batch_variant_info(int v, int* threads, int* ctas_per_sm)
{
    if (v < 0 || v >= kNumBatchVariants || !threads || !ctas_per_sm) return CLAW2_ERR_INVALID;
    *threads = kBatchVariants[v].threads;
    *ctas_per_sm = kBatchVariants[v].minb;
    return CLAW2_OK;
}

int claw2_batch_tiles(int mx, int my, int* nbx, int* nby)
{
    return claw2_batch_tiles_for(29, mx, my, nbx, nby);
}

int claw2_batch_variant_tile(int v)
{
    if (v < 0 || v >= kNumBatchVariants) return -1;
    return kBatchVariants[v].tile;
}

int claw2_batch_tiles_for(int tile, int mx, int my, int* nbx, int* nby)
{
    if (!batch_tile_ok(tile) || mx < 4 || my < 4 || !nbx || !nby) return CLAW2_ERR_INVALID;
    const int width = batch_march_tile(tile) ? MARCH_TX : tile;
    *nbx = (mx + width - 1) / width;
    *nby = (my + tile - 1) / tile;
    return CLAW2_OK;
}

int claw2_batch_advance(const claw2_problem* p, const claw2_batch_instance* inst, int ninst, int ntiles, int nsteps,
                        int variant, void* stream)
{
    return claw2_batch_advance_map(p, inst, ninst, ntiles, nullptr, nsteps, variant, stream);
}

int claw2_batch_advance_map(const claw2_problem* p, const claw2_batch_instance* inst, int ninst, int ntiles,
                            const int32_t* tile_inst, int nsteps, int variant, void* stream)
{
    int rc = batch_check(p, inst, ninst, ntiles, nsteps, variant);
    if (rc) return rc;
    return batch_launch(p, inst, ninst, ntiles, nsteps, variant, tile_inst, S(stream));
}

int claw2_batch_graph_create(const claw2_problem* p, const claw2_batch_instance* inst, int ninst, int ntiles,
                             int nsteps, int variant, void** graph_exec)
{
    return claw2_batch_graph_create_map(p, inst, ninst, ntiles, nullptr, nsteps, variant, graph_exec);
}

int claw2_batch_graph_create_map(const claw2_problem* p, const claw2_batch_instance* inst, int ninst, int ntiles,
                                 const int32_t* tile_inst, int nsteps, int variant, void** graph_exec)
{
    int rc = batch_check(p, inst, ninst, ntiles, nsteps, variant);
    if (rc) return rc;
    if (!graph_exec) return CLAW2_ERR_INVALID;
    // one launch outside the capture configures the kernel (shared-memory
    // attribute, occupancy) so that the capture itself only records launches
    cudaStream_t st;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return CLAW2_ERR_CUDA;
    rc = batch_launch(p, inst, ninst, ntiles, 0, variant, tile_inst, st);
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    if (!rc && cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) rc = CLAW2_ERR_CUDA;
    if (!rc) {
        const int r2 = batch_launch(p, inst, ninst, ntiles, nsteps, variant, tile_inst, st);
        if (cudaStreamEndCapture(st, &graph) != cudaSuccess || r2) rc = r2 ? r2 : CLAW2_ERR_CUDA;
    }
    if (!rc && cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) rc = CLAW2_ERR_CUDA;
    if (graph) cudaGraphDestroy(graph);
    cudaStreamDestroy(st);
    if (rc) return rc;
    *graph_exec = exec;
    return CLAW2_OK;
}

}  // extern "C"
