// claw2_capi.cu -- CUDA kernels and the extern "C" ABI declared in include/claw2.h.
//
// Built for sm_100a with --fmad=false (no FMA contraction, so the step
// reproduces the reference's operation-by-operation rounding).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <new>

#define CLAW2_EXPORT __attribute__((visibility("default")))
#include "../../include/claw2.h"
#include "claw2_devattr.h"
#include "claw2_host.h"
#include "claw2_kernels.cuh"
#include "claw2_launch.cuh"

namespace claw2 {

#ifndef CLAW2_MINB
#define CLAW2_MINB 2        // resident CTAs per SM the register budget is sized for
#endif

template <class RP, int TX, int TY, int NT, bool SPLIT>
__global__ void __launch_bounds__(NT, CLAW2_MINB) step_kernel(StepArgs a)
{
    chain_wait();
    extern __shared__ double smem_dyn[];
    DevCtx ctx{smem_dyn};
    step_tile<RP, TX, TY, NT, SPLIT>(a, ctx);
}

// Tile shapes: a line of a chunk has 32 interface slots, so TX+3, TY+3 <= 32.
#ifndef CLAW2_UNT
#define CLAW2_UNT 256
#endif
constexpr int UTX = 29, UTY = 29, UNT = CLAW2_UNT;   // unsplit
constexpr int STX = 28, STY = 28, SNT = 256;   // dimensional splitting

// ---------------------------------------------------------------------------
// ghost fill (device layout): Solver.apply_q_bcs, x sides then y sides
// ---------------------------------------------------------------------------
struct FillArgs {
    double* q;
    long long ld, plane;
    int mx, my, ncomp;
    int bl, bu;        // this axis' lower/upper BC
    int negate;        // 0-based component negated at walls (-1 none)
};

// axis 0 fills ghost columns over all rows (incl. ghost rows); axis 1 fills ghost
// rows over all columns.  One thread per (component, position along the other
// axis, ghost layer, side).
template <int AXIS>
__device__ __forceinline__ void fill_body(const FillArgs& f)
{
    const int other = (AXIS == 0 ? f.my : f.mx) + 2 * CLAW2_NUM_GHOST;
    const int n = AXIS == 0 ? f.mx : f.my;
    const long long total = (long long)f.ncomp * other * 2 * CLAW2_NUM_GHOST;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
        const int o = (int)(t % other) - CLAW2_NUM_GHOST;
        long long r = t / other;
        const int g = (int)(r % CLAW2_NUM_GHOST);
        r /= CLAW2_NUM_GHOST;
        const int side = (int)(r % 2);
        const int m = (int)(r / 2);
        const int bc = side == 0 ? f.bl : f.bu;
        int dst, src;
        if (side == 0) {
            dst = -1 - g;
            if (bc == CLAW2_BC_EXTRAP) src = 0;
            else if (bc == CLAW2_BC_PERIODIC) src = n - 1 - g;
            else if (bc == CLAW2_BC_WALL) src = g;
            else continue;
        } else {
            dst = n + g;
            if (bc == CLAW2_BC_EXTRAP) src = n - 1;
            else if (bc == CLAW2_BC_PERIODIC) src = g;
            else if (bc == CLAW2_BC_WALL) src = n - 1 - g;
            else continue;
        }
        auto off = [&](int along) {
            const int i = AXIS == 0 ? along : o, j = AXIS == 0 ? o : along;
            return (long long)m * f.plane + (long long)(j + CLAW2_NUM_GHOST) * f.ld + (i + CLAW2_NUM_GHOST);
        };
        double v = f.q[off(src)];
        if (bc == CLAW2_BC_WALL && m == f.negate) v = -v;
        f.q[off(dst)] = v;
    }
}

template <int AXIS>
__global__ void fill_kernel(FillArgs f)
{
    fill_body<AXIS>(f);
}

// Fill the ghost cells of q[ctrl->cur] (used after controlled steps when the
// step kernel cannot write ghost images itself).
template <int AXIS>
__global__ void fill_kernel_ctrl(FillArgs f, double* q0, double* q1, const claw2_control* c)
{
    f.q = c->cur ? q1 : q0;
    fill_body<AXIS>(f);
}

// ---------------------------------------------------------------------------
// layout conversion: reference (m fastest, Fortran) <-> device (planes)
// ---------------------------------------------------------------------------
// A thread per cell and its nc components (a thread per element spent most of its time
// on two 64-bit divisions: 320 x 160 Euler session step with both copies 117 -> 111 us
// together with the launches as programmatic dependents).
constexpr int CONV_NT = 128;

__global__ void __launch_bounds__(CONV_NT) ref_to_dev_kernel(const double* ref, double* dev, int nc, int nx, int ny,
                                                             long long ld, long long plane, int off)
{
    chain_wait();
    const int i = blockIdx.x * CONV_NT + threadIdx.x;
    if (i >= nx) return;
    for (int j = blockIdx.y; j < ny; j += gridDim.y) {
        const double* r = ref + ((long long)j * nx + i) * nc;
        double* d = dev + (long long)(j + off) * ld + (i + off);
        for (int m = 0; m < nc; m++) d[m * plane] = r[m];
    }
}

__global__ void __launch_bounds__(CONV_NT) dev_to_ref_kernel(const double* dev, double* ref, int nc, int nx, int ny,
                                                             long long ld, long long plane, int off)
{
    chain_wait();
    const int i = blockIdx.x * CONV_NT + threadIdx.x;
    if (i >= nx) return;
    for (int j = blockIdx.y; j < ny; j += gridDim.y) {
        double* r = ref + ((long long)j * nx + i) * nc;
        const double* d = dev + (long long)(j + off) * ld + (i + off);
        for (int m = 0; m < nc; m++) r[m] = d[m * plane];
    }
}

// domain decomposition helpers: controller update from a given CFL number,
// and the two halo rows of q[cur] to/from a contiguous buffer
__global__ void control_apply_kernel(claw2_control* c, const double* cfl)
{
    const double v = *cfl;
    const bool nonfinite = !(v < 1.0 / 0.0);          // +inf or NaN
    if (!c->done) control_update(c, nonfinite ? 0.0 : v, nonfinite ? 1 : 0);
}

__global__ void halo_kernel(double* q0, double* q1, const claw2_control* c, double* buf, long long ld,
                            long long plane, int mx, int my, int ncomp, int upper, int unpack)
{
    double* q = c->cur ? q1 : q0;
    const int w = mx + 2 * CLAW2_NUM_GHOST;
    const int total = ncomp * 2 * w;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const int i = t % w - CLAW2_NUM_GHOST, r = (t / w) % 2, m = t / (2 * w);
        int row;
        if (!unpack) row = upper ? my - 2 + r : r;
        else row = upper ? my + r : -2 + r;
        const long long o = (long long)m * plane + (long long)(row + CLAW2_NUM_GHOST) * ld + (i + CLAW2_NUM_GHOST);
        if (unpack) q[o] = buf[t];
        else buf[t] = q[o];
    }
}

// Before-step copy of plane `from` of q[cur] (ghost cells included) into
// plane `to` of aux (claw2_hooks.aux_from_q).
__global__ void aux_from_q_kernel(double* aux, const double* q0, const double* q1, const claw2_control* c,
                                  long long plane, int from, int to)
{
    chain_wait();
    if (c->done) return;
    const double* q = (c->cur ? q1 : q0) + (long long)from * plane;
    double* d = aux + (long long)to * plane;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < plane; t += (long long)gridDim.x * blockDim.x)
        d[t] = q[t];
}

// Gauge samples after a step (claw2_gauges): one block; nothing happens
// unless the controller accepted a step since the last row.
__global__ void gauge_record_kernel(claw2_gauges g, const double* q0, const double* q1, const claw2_control* c,
                                    int meqn, long long ld, long long plane, int mx, int my)
{
    __shared__ int row;
    chain_wait();
    if (threadIdx.x == 0) {
        row = -1;
        if (c->numsteps != g.state[1]) {
            if (g.state[0] < g.capacity) row = (int)g.state[0];
            else g.state[2] = 1;
        }
    }
    __syncthreads();
    if (row < 0) return;
    const double* q = c->cur ? q1 : q0;
    const int w = 1 + meqn;
    for (int idx = threadIdx.x; idx < g.ngauges * w; idx += blockDim.x) {
        const int k = idx / w, m = idx - k * w;
        double v;
        if (m == 0) v = c->t;
        else {
            const int ix = g.cells[2 * k], iy = g.cells[2 * k + 1];
            if (ix < 0 || ix >= mx || iy < 0 || iy >= my) v = __longlong_as_double(0x7ff8000000000000ULL);
            else v = q[(long long)(m - 1) * plane + (long long)(iy + CLAW2_NUM_GHOST) * ld + ix + CLAW2_NUM_GHOST];
        }
        g.record[((long long)row * g.ngauges + k) * w + m] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        g.state[0] = row + 1;
        g.state[1] = c->numsteps;
    }
}

}  // namespace claw2

using namespace claw2;

// ===========================================================================
// host helpers
// ===========================================================================
namespace {

// Problems stepped by the marching body, split by the row body (launch_step): the
// acoustics solvers without capacity or f-waves.
bool march_body(const claw2_problem* p)
{
    return p->index_capa < 0 && !p->use_fwave &&
           (p->rp == CLAW2_RP_ACOUSTICS || p->rp == CLAW2_RP_VC_ACOUSTICS);
}

// Problems stepped by the lean body (launch_step): Euler and shallow water
// without capacity or f-waves.
bool lean_body(const claw2_problem* p)
{
    return p->index_capa < 0 && !p->use_fwave &&
           (p->rp == CLAW2_RP_EULER_4WAVE || p->rp == CLAW2_RP_EULER_5WAVE || p->rp == CLAW2_RP_SHALLOW_ROE);
}

// Arguments of a step whose ghost cells the caller does not fill himself: beside
// custom sides the tile bodies write them too (the marching body does not).
void step_args(const claw2_problem* p, double* q, StepArgs& a)
{
    fill_args(p, q, a);
    if (!a.ghost_fused && fused_beside_custom(p) && !(march_body(p) && p->transverse >= 0)) a.ghost_fused = a.custom = 1;
}

// The tiles that claw2_scratch_bytes counts for it: 29x29 cells, 13x13 on
// grids of fewer than 148 such tiles.  No kernel has them: like the split acoustics and
// the p-system bodies, this one needs the header alone.  The count stays, and with it
// the scratch size and claw2_step_noalloc's largest grid, as callers know them.
constexpr int MARCH_SMALL_TILE = 13;
bool march_small_grid(int mx, int my)
{
    return (long long)((mx + 28) / 29) * (long long)((my + 28) / 29) < 148;
}

void tiles(const claw2_problem* p, int* nbx, int* nby)
{
    const bool split = p->transverse < 0;
    int tx = split ? STX : UTX, ty = split ? STY : UTY;
    // (for the scratch size alone)
    if (!split && march_body(p) && march_small_grid(p->mx, p->my)) tx = ty = MARCH_SMALL_TILE;
    // the lean body lists its 28-tiles in the scratch
    if (lean_body(p)) tx = ty = LEAN_T;
    *nbx = (p->mx + tx - 1) / tx;
    *nby = (p->my + ty - 1) / ty;
}

// The scratch of a step: the 64-byte header (arrival counter, CFL maximum, number of
// listed tiles) and eight bytes per tile (the generic body's CFL partials, the lean
// body's list).
size_t scratch_bytes(const claw2_problem* p)
{
    int nbx, nby;
    tiles(p, &nbx, &nby);
    return 64 + sizeof(double) * (size_t)nbx * (size_t)nby;
}

// Point a's arrival counter and partials into scratch.
void set_scratch(void* scratch, StepArgs& a)
{
    a.ticket = static_cast<unsigned int*>(scratch);
    a.partials = reinterpret_cast<double*>(static_cast<char*>(scratch) + 64);
}

// bytes of halo that lean-body CTAs wait for in vain (claw2_debug_halo_shortfall)
std::atomic<int> g_halo_shortfall{0};

template <class RP, bool SPLIT>
int launch_step_t(const StepArgs& a, int nbx, int nby, cudaStream_t st, bool chained)
{
    constexpr int TX = SPLIT ? STX : UTX, TY = SPLIT ? STY : UTY, NT = SPLIT ? SNT : UNT;
    using SM = TileSmem<RP, TX, TY, NT, SPLIT>;
    auto kern = step_kernel<RP, TX, TY, NT, SPLIT>;
    static std::atomic<uint64_t> optin{0};
    if (smem_optin(optin, kern, SM::bytes) != cudaSuccess) return CLAW2_ERR_CUDA;
    return launch_kernel(kern, dim3(nbx, nby), NT, SM::bytes, st, chained, a);
}

// chained: the previous operation in the stream is a step kernel of the same
// device loop, so this step may overlap its end (launch_kernel).
int launch_step(const claw2_problem* p, const StepArgs& a, cudaStream_t st, bool chained = false)
{
    const bool split = p->transverse < 0;
    if (march_body(p)) return split ? launch_rows(p->rp, a, st, chained) : launch_march(p->rp, a, st, chained);
    if (p->rp == CLAW2_RP_PSYSTEM && p->use_fwave && p->index_capa < 0 && !split) return launch_psystem(a, st, chained);
    // the lean body's halo copies start on 16-byte boundaries; other buffers keep
    // the general split body (unsplit they are refused)
    const uintptr_t start = a.ctrl ? reinterpret_cast<uintptr_t>(a.q0) | reinterpret_cast<uintptr_t>(a.q1)
                                   : reinterpret_cast<uintptr_t>(a.qin);
    if (lean_body(p) && (!split || (start & 15u) == 0)) {
        StepArgs l = a;
        l.halo_shortfall = g_halo_shortfall.load(std::memory_order_relaxed);
        return launch_lean(p->rp, split, l, st, chained);
    }
    int nbx, nby;
    tiles(p, &nbx, &nby);
    switch (p->rp) {
    case CLAW2_RP_ACOUSTICS:
        return split ? launch_step_t<RpAcoustics, true>(a, nbx, nby, st, chained) : launch_step_t<RpAcoustics, false>(a, nbx, nby, st, chained);
    case CLAW2_RP_VC_ACOUSTICS:
        return split ? launch_step_t<RpVcAcoustics, true>(a, nbx, nby, st, chained) : launch_step_t<RpVcAcoustics, false>(a, nbx, nby, st, chained);
    case CLAW2_RP_EULER_4WAVE:
        return split ? launch_step_t<RpEuler<false>, true>(a, nbx, nby, st, chained) : launch_step_t<RpEuler<false>, false>(a, nbx, nby, st, chained);
    case CLAW2_RP_EULER_5WAVE:
        return split ? launch_step_t<RpEuler<true>, true>(a, nbx, nby, st, chained) : launch_step_t<RpEuler<true>, false>(a, nbx, nby, st, chained);
    case CLAW2_RP_SHALLOW_ROE:
        return split ? launch_step_t<RpShallow, true>(a, nbx, nby, st, chained) : launch_step_t<RpShallow, false>(a, nbx, nby, st, chained);
    case CLAW2_RP_PSYSTEM:
        return split ? launch_step_t<RpPsystem, true>(a, nbx, nby, st, chained) : launch_step_t<RpPsystem, false>(a, nbx, nby, st, chained);
    default:
        return CLAW2_ERR_INVALID;
    }
}

int launch_fill(const claw2_problem* p, double* q, int ncomp, const int* bl, const int* bu, bool is_aux,
                double* q0, double* q1, const claw2_control* ctrl, cudaStream_t st)
{
    claw2_layout L;
    claw2_get_layout(p, &L);
    for (int axis = 0; axis < 2; axis++) {
        FillArgs f;
        f.q = q; f.ld = L.ld; f.plane = L.plane; f.mx = p->mx; f.my = p->my; f.ncomp = ncomp;
        f.bl = bl[axis]; f.bu = bu[axis];
        f.negate = is_aux ? -1 : axis + 1;
        const int other = (axis == 0 ? p->my : p->mx) + 2 * CLAW2_NUM_GHOST;
        const long long total = (long long)ncomp * other * 2 * CLAW2_NUM_GHOST;
        const int threads = 256;
        const int blocks = (int)((total + threads - 1) / threads);
        if (ctrl) {
            if (axis == 0) fill_kernel_ctrl<0><<<blocks, threads, 0, st>>>(f, q0, q1, ctrl);
            else fill_kernel_ctrl<1><<<blocks, threads, 0, st>>>(f, q0, q1, ctrl);
        } else {
            if (axis == 0) fill_kernel<0><<<blocks, threads, 0, st>>>(f);
            else fill_kernel<1><<<blocks, threads, 0, st>>>(f);
        }
        if (cudaGetLastError() != cudaSuccess) return CLAW2_ERR_CUDA;
    }
    return CLAW2_OK;
}

// chained: the previous operation in the stream is a step kernel of the same call.
int conv(const claw2_problem* p, int ncomp, const double* src, double* dst, bool to_dev, bool ghosts, cudaStream_t st,
         bool chained = false)
{
    claw2_layout L;
    int rc = claw2_get_layout(p, &L);
    if (rc) return rc;
    const int g = ghosts ? 2 * CLAW2_NUM_GHOST : 0, off = ghosts ? 0 : CLAW2_NUM_GHOST;
    const int nx = p->mx + g, ny = p->my + g;
    const dim3 grid((nx + CONV_NT - 1) / CONV_NT, ny < 65535 ? ny : 65535);
    return launch_kernel(to_dev ? ref_to_dev_kernel : dev_to_ref_kernel, grid, CONV_NT, 0, st, chained, src, dst, ncomp, nx, ny,
                         (long long)L.ld, (long long)L.plane, off);
}

}  // namespace

// ===========================================================================
// extern "C" ABI
// ===========================================================================
extern "C" {

int claw2_abi_version(void) { return CLAW2_ABI_VERSION; }

int claw2_debug_halo_shortfall(int bytes)
{
    if (bytes < 0 || bytes > 65536 || (bytes & 7)) return CLAW2_ERR_INVALID;
    g_halo_shortfall.store(bytes, std::memory_order_relaxed);
    return CLAW2_OK;
}

const char* claw2_strerror(int status)
{
    switch (status) {
    case CLAW2_OK: return "ok";
    case CLAW2_ERR_INVALID: return "invalid problem description or argument";
    case CLAW2_ERR_UNSUPPORTED: return "feature not supported by this build";
    case CLAW2_ERR_CUDA: return "CUDA runtime error";
    case CLAW2_ERR_CFL: return "CFL too large, giving up!";
    case CLAW2_ERR_MAX_STEPS: return "Maximum number of timesteps have been taken";
    case CLAW2_ERR_NONFINITE: return "non-finite or non-physical state produced";
    case CLAW2_ERR_TIMEOUT: return "bounded device wait gave up";
    case CLAW2_ERR_NOMEM: return "out of memory";
    case CLAW2_ERR_SIZE: return "size beyond the documented maximum";
    default: return "unknown claw2 status";
    }
}

int claw2_validate(const claw2_problem* p)
{
    int meqn, mw, maux;
    if (!p) return CLAW2_ERR_INVALID;
    if (solver_shape(p->rp, &meqn, &mw, &maux)) return CLAW2_ERR_INVALID;
    if (p->num_eqn != meqn || p->num_waves != mw || p->num_aux < maux) return CLAW2_ERR_INVALID;
    if (p->num_ghost != CLAW2_NUM_GHOST) return CLAW2_ERR_UNSUPPORTED;
    if (p->mx < 2 || p->my < 2) return CLAW2_ERR_INVALID;
    if (p->num_aux < 0 || p->num_aux > CLAW2_MAX_EQN) return CLAW2_ERR_INVALID;
    if (p->order < 1 || p->order > 2) return CLAW2_ERR_INVALID;
    if (p->transverse < -1 || p->transverse > 2) return CLAW2_ERR_INVALID;
    if (p->index_capa < -1 || p->index_capa >= p->num_aux) return CLAW2_ERR_INVALID;
    if (!(p->dx > 0.0) || !(p->dy > 0.0)) return CLAW2_ERR_INVALID;
    for (int w = 0; w < p->num_waves; w++)
        if (p->mthlim[w] < 0) return CLAW2_ERR_INVALID;
    for (int d = 0; d < 2; d++) {
        if (p->bc_lower[d] < 0 || p->bc_lower[d] > 3 || p->bc_upper[d] < 0 || p->bc_upper[d] > 3) return CLAW2_ERR_INVALID;
        if (!periodic_ok(p->bc_lower[d], p->bc_upper[d])) return CLAW2_ERR_UNSUPPORTED;
        if (p->num_aux > 0 && (p->aux_bc_lower[d] < 0 || p->aux_bc_lower[d] > 3 ||
                               p->aux_bc_upper[d] < 0 || p->aux_bc_upper[d] > 3)) return CLAW2_ERR_INVALID;
    }
    return CLAW2_OK;
}

int claw2_get_layout(const claw2_problem* p, claw2_layout* out)
{
    if (!p || !out || p->mx < 1 || p->my < 1) return CLAW2_ERR_INVALID;
    const long long nx = (long long)p->mx + 2 * CLAW2_NUM_GHOST;
    out->ld = (nx + 15) / 16 * 16;              // 128-byte row pitch
    out->rows = (long long)p->my + 2 * CLAW2_NUM_GHOST;
    out->plane = out->ld * out->rows;
    out->q_elems = (long long)p->num_eqn * out->plane;
    out->aux_elems = (long long)p->num_aux * out->plane;
    return CLAW2_OK;
}

size_t claw2_scratch_bytes(const claw2_problem* p)
{
    if (!p || p->mx < 1 || p->my < 1) return 0;
    return scratch_bytes(p);
}

int claw2_fill_ghosts(const claw2_problem* p, double* q, void* stream)
{
    int rc = claw2_validate(p);
    if (rc) return rc;
    return launch_fill(p, q, p->num_eqn, p->bc_lower, p->bc_upper, false, nullptr, nullptr, nullptr, S(stream));
}

int claw2_fill_aux_ghosts(const claw2_problem* p, double* aux, void* stream)
{
    int rc = claw2_validate(p);
    if (rc) return rc;
    if (p->num_aux == 0) return CLAW2_OK;
    return launch_fill(p, aux, p->num_aux, p->aux_bc_lower, p->aux_bc_upper, true, nullptr, nullptr, nullptr, S(stream));
}

}  // extern "C"

namespace {
// claw2_step.  chained: the previous operation in the stream is a conversion kernel
// (conv).  *last: whether its last operation is a step kernel.
int step_once(const claw2_problem* p, const double* q_in, double* q_out, const double* aux, double dt, void* scratch,
              double* cfl_dev, void* stream, bool chained, bool* last)
{
    int rc = claw2_validate(p);
    if (rc) return rc;
    if (!q_in || !q_out || !scratch || !cfl_dev || (p->num_aux > 0 && !aux) || q_in == q_out) return CLAW2_ERR_INVALID;
    StepArgs a;
    step_args(p, q_out, a);
    if (last) *last = a.ghost_fused != 0;
    a.qin = q_in; a.qout = q_out; a.aux = aux; a.dt = dt;
    set_scratch(scratch, a);
    a.cfl_out = cfl_dev;
    if ((rc = launch_step(p, a, S(stream), chained))) return rc;
    if (!a.ghost_fused)
        return launch_fill(p, q_out, p->num_eqn, p->bc_lower, p->bc_upper, false, nullptr, nullptr, nullptr, S(stream));
    return CLAW2_OK;
}
}  // namespace

extern "C" {

int claw2_step(const claw2_problem* p, const double* q_in, double* q_out, const double* aux, double dt,
               void* scratch, double* cfl_dev, void* stream)
{
    return step_once(p, q_in, q_out, aux, dt, scratch, cfl_dev, stream, false, nullptr);
}

int claw2_advance(const claw2_problem* p, double* q0, double* q1, const double* aux, claw2_control* ctrl,
                  void* scratch, int nsteps, void* stream)
{
    int rc = claw2_validate(p);
    if (rc) return rc;
    if (!q0 || !q1 || !ctrl || !scratch || (p->num_aux > 0 && !aux) || nsteps < 0) return CLAW2_ERR_INVALID;
    StepArgs a;
    step_args(p, q0, a);
    a.q0 = q0; a.q1 = q1; a.aux = aux; a.ctrl = ctrl;
    set_scratch(scratch, a);
    for (int n = 0; n < nsteps; n++) {
        // from the second step on, a step follows a step kernel directly
        if ((rc = launch_step(p, a, S(stream), n > 0 && a.ghost_fused))) return rc;
        if (!a.ghost_fused &&
            (rc = launch_fill(p, nullptr, p->num_eqn, p->bc_lower, p->bc_upper, false, q0, q1, ctrl, S(stream))))
            return rc;
    }
    return CLAW2_OK;
}

}  // extern "C"

namespace {
// Checks claw2_hooks against the problem and sets the source term in a.
int apply_hooks(const claw2_problem* p, const claw2_hooks* hooks, StepArgs& a)
{
    if (hooks->source != CLAW2_SRC_NONE && hooks->source != CLAW2_SRC_EULER_RADIAL) return CLAW2_ERR_INVALID;
    if (hooks->source == CLAW2_SRC_EULER_RADIAL &&
        ((p->rp != CLAW2_RP_EULER_4WAVE && p->rp != CLAW2_RP_EULER_5WAVE) || hooks->source_aux < 0 ||
         hooks->source_aux >= p->num_aux))
        return CLAW2_ERR_UNSUPPORTED;
    if (hooks->aux_from_q != 0) {
        const int k = hooks->aux_from_q - 1, m = hooks->aux_q - 1;
        if (k < 0 || k >= p->num_aux || m < 0 || m >= p->num_eqn) return CLAW2_ERR_INVALID;
        for (int d = 0; d < 2; d++)
            if (p->aux_bc_lower[d] != p->bc_lower[d] || p->aux_bc_upper[d] != p->bc_upper[d] ||
                p->bc_lower[d] == CLAW2_BC_CUSTOM || p->bc_upper[d] == CLAW2_BC_CUSTOM)
                return CLAW2_ERR_UNSUPPORTED;
    }
    a.src = hooks->source;
    a.src_aux = hooks->source_aux;
    return CLAW2_OK;
}

// One step of a loop with hooks (or gauges, hooks null then).  chained: the previous
// operation in the stream is a step or gauge kernel of the same loop; the kernels here
// wait for the one before them themselves (chain_wait).
int launch_hooked(const claw2_problem* p, const claw2_hooks* hooks, const StepArgs& a, double* aux, bool chained,
                  cudaStream_t st)
{
    int rc;
    if (hooks && hooks->aux_from_q != 0) {
        int blocks = (int)((a.plane + 255) / 256);
        if (blocks > 148 * 8) blocks = 148 * 8;
        if ((rc = launch_kernel(aux_from_q_kernel, dim3(blocks), 256, 0, st, chained, aux, (const double*)a.q0,
                                (const double*)a.q1, (const claw2_control*)a.ctrl, a.plane, hooks->aux_q - 1,
                                hooks->aux_from_q - 1)))
            return rc;
        chained = true;
    }
    if ((rc = launch_step(p, a, st, chained)) || a.ghost_fused) return rc;
    return launch_fill(p, nullptr, p->num_eqn, p->bc_lower, p->bc_upper, false, a.q0, a.q1, a.ctrl, st);
}
}  // namespace

extern "C" {

int claw2_advance_hooked(const claw2_problem* p, double* q0, double* q1, const double* aux, claw2_control* ctrl,
                         void* scratch, int nsteps, const claw2_hooks* hooks, void* stream)
{
    int rc = claw2_validate(p);
    if (rc) return rc;
    if (!q0 || !q1 || !ctrl || !scratch || !hooks || (p->num_aux > 0 && !aux) || nsteps < 0) return CLAW2_ERR_INVALID;
    StepArgs a;
    step_args(p, q0, a);
    a.q0 = q0; a.q1 = q1; a.aux = aux; a.ctrl = ctrl;
    set_scratch(scratch, a);
    if ((rc = apply_hooks(p, hooks, a))) return rc;
    for (int n = 0; n < nsteps; n++)
        if ((rc = launch_hooked(p, hooks, a, const_cast<double*>(aux), n > 0 && a.ghost_fused, S(stream)))) return rc;
    return CLAW2_OK;
}

int claw2_advance_gauged(const claw2_problem* p, double* q0, double* q1, const double* aux, claw2_control* ctrl,
                         void* scratch, int nsteps, const claw2_hooks* hooks, const claw2_gauges* g, void* stream)
{
    int rc = claw2_validate(p);
    if (rc) return rc;
    if (!q0 || !q1 || !ctrl || !scratch || !g || (p->num_aux > 0 && !aux) || nsteps < 0) return CLAW2_ERR_INVALID;
    if (g->ngauges < 1 || g->capacity < 1 || !g->cells || !g->record || !g->state) return CLAW2_ERR_INVALID;
    StepArgs a;
    step_args(p, q0, a);
    a.q0 = q0; a.q1 = q1; a.aux = aux; a.ctrl = ctrl;
    set_scratch(scratch, a);
    if (hooks && (rc = apply_hooks(p, hooks, a))) return rc;
    const int threads = 128;
    for (int n = 0; n < nsteps; n++) {
        if ((rc = launch_hooked(p, hooks, a, const_cast<double*>(aux), n > 0, S(stream)))) return rc;
        if ((rc = launch_kernel(gauge_record_kernel, dim3(1), threads, 0, S(stream), a.ghost_fused, *g,
                                (const double*)q0, (const double*)q1, (const claw2_control*)ctrl, (int)p->num_eqn, a.ld, a.plane,
                                (int)p->mx, (int)p->my)))
            return rc;
    }
    return CLAW2_OK;
}

int claw2_step_ctrl(const claw2_problem* p, double* q0, double* q1, const double* aux, claw2_control* ctrl,
                    void* scratch, double* cfl_dev, void* stream)
{
    int rc = claw2_validate(p);
    if (rc) return rc;
    if (!q0 || !q1 || !ctrl || !scratch || !cfl_dev || (p->num_aux > 0 && !aux)) return CLAW2_ERR_INVALID;
    StepArgs a;
    fill_args(p, q0, a);
    a.q0 = q0; a.q1 = q1; a.aux = aux; a.ctrl = ctrl;
    a.ctrl_readonly = 1;
    a.cfl_out = cfl_dev;
    a.ghost_fused = 0;
    set_scratch(scratch, a);
    return launch_step(p, a, S(stream));
}

int claw2_control_apply(claw2_control* ctrl, const double* cfl_dev, void* stream)
{
    if (!ctrl || !cfl_dev) return CLAW2_ERR_INVALID;
    control_apply_kernel<<<1, 1, 0, S(stream)>>>(ctrl, cfl_dev);
    return cudaGetLastError() == cudaSuccess ? CLAW2_OK : CLAW2_ERR_CUDA;
}

int claw2_fill_ghosts_ctrl(const claw2_problem* p, double* q0, double* q1, const claw2_control* ctrl, void* stream)
{
    int rc = claw2_validate(p);
    if (rc) return rc;
    if (!q0 || !q1 || !ctrl) return CLAW2_ERR_INVALID;
    return launch_fill(p, nullptr, p->num_eqn, p->bc_lower, p->bc_upper, false, q0, q1, ctrl, S(stream));
}

static int halo(const claw2_problem* p, double* q0, double* q1, const claw2_control* ctrl, int upper, double* buf,
                int unpack, void* stream)
{
    int rc = claw2_validate(p);
    if (rc) return rc;
    if (!q0 || !q1 || !ctrl || !buf || (upper != 0 && upper != 1) || p->my < 2) return CLAW2_ERR_INVALID;
    claw2_layout L;
    claw2_get_layout(p, &L);
    const int total = p->num_eqn * 2 * (p->mx + 2 * CLAW2_NUM_GHOST);
    halo_kernel<<<(total + 255) / 256, 256, 0, S(stream)>>>(q0, q1, ctrl, buf, L.ld, L.plane, p->mx, p->my,
                                                           p->num_eqn, upper, unpack);
    return cudaGetLastError() == cudaSuccess ? CLAW2_OK : CLAW2_ERR_CUDA;
}

int claw2_halo_pack(const claw2_problem* p, const double* q0, const double* q1, const claw2_control* ctrl, int upper,
                    double* buf, void* stream)
{
    return halo(p, const_cast<double*>(q0), const_cast<double*>(q1), ctrl, upper, buf, 0, stream);
}

int claw2_halo_unpack(const claw2_problem* p, double* q0, double* q1, const claw2_control* ctrl, int upper,
                      const double* buf, void* stream)
{
    return halo(p, q0, q1, ctrl, upper, const_cast<double*>(buf), 1, stream);
}

int claw2_control_init(claw2_control* c, double t, double dt, double tend, double cfl_max, double cfl_desired,
                       double dt_max, int dt_variable, int take_one_step, int64_t max_steps, double prev_cfl)
{
    if (!c) return CLAW2_ERR_INVALID;
    std::memset(c, 0, sizeof *c);
    c->t = t; c->dt = dt; c->tstart = t; c->tend = tend;
    c->cfl = prev_cfl;
    c->cfl_max = cfl_max; c->cfl_desired = cfl_desired; c->dt_max = dt_max;
    c->status_cflmax = prev_cfl; c->status_dtmin = dt; c->status_dtmax = dt;
    c->dt_variable = dt_variable; c->take_one_step = take_one_step;
    c->max_steps = max_steps;
    if (!dt_variable) {                                       // solver.py:618-624
        if (take_one_step) c->max_steps = 1;
        else {
            c->max_steps = (int64_t)((tend - t + 1e-10) / dt);
            if (std::fabs(c->max_steps * dt - (tend - t)) > 1e-5 * (tend - t)) return CLAW2_ERR_INVALID;
        }
    }
    if (dt_variable && cfl_desired > cfl_max) return CLAW2_ERR_INVALID;   // :625-626
    if (tend <= t && !take_one_step) c->max_steps = 0;                     // :627-629
    if (c->max_steps <= 0) { c->done = 1; return CLAW2_OK; }
    if (!take_one_step) {                                                  // :637-641
        if (c->t + c->dt > c->tend && c->tstart < c->tend) c->dt = c->tend - c->t;
        if (c->tend - c->t - c->dt < 1.e-14 * c->t) c->dt = c->tend - c->t;
    }
    return CLAW2_OK;
}

int claw2_ref_to_device(const claw2_problem* p, int ncomp, const double* ref, double* dev, void* stream)
{
    if (!p || !ref || !dev || ncomp < 1) return CLAW2_ERR_INVALID;
    return conv(p, ncomp, ref, dev, true, true, S(stream));
}

int claw2_device_to_ref(const claw2_problem* p, int ncomp, const double* dev, double* ref, void* stream)
{
    if (!p || !ref || !dev || ncomp < 1) return CLAW2_ERR_INVALID;
    return conv(p, ncomp, dev, ref, false, true, S(stream));
}

int claw2_graph_launch(void* graph_exec, void* stream)
{
    if (!graph_exec) return CLAW2_ERR_INVALID;
    return cudaGraphLaunch(reinterpret_cast<cudaGraphExec_t>(graph_exec), S(stream)) == cudaSuccess ? CLAW2_OK
                                                                                                     : CLAW2_ERR_CUDA;
}

int claw2_graph_destroy(void* graph_exec)
{
    if (!graph_exec) return CLAW2_OK;
    return cudaGraphExecDestroy(reinterpret_cast<cudaGraphExec_t>(graph_exec)) == cudaSuccess ? CLAW2_OK
                                                                                               : CLAW2_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// allocation-free step
//
// Some callers cannot allocate GPU memory: a host code that hands all device
// memory to its own pool at start-up, a time loop that must not enter the CUDA
// allocator (an allocation can synchronise the device), or a foreign-language
// binding that can pass pointers to existing buffers but cannot own device
// allocations.  claw2_step_noalloc serves them: its scratch (the header and
// eight bytes per tile, as claw2_scratch_bytes) is the static array below, which every
// GPU that loads this library holds until the process exits.
// ---------------------------------------------------------------------------
}  // extern "C"

static __device__ __align__(256) unsigned char g_noalloc_scratch[64 + 8 * CLAW2_NOALLOC_MAX_TILES];

namespace {
constexpr int kMaxDevices = 64;
std::atomic<void*> g_noalloc_addr[kMaxDevices];   // device address of g_noalloc_scratch, per device
}

extern "C" {

int claw2_step_noalloc(const claw2_problem* p, const double* q_in, double* q_out, const double* aux, double dt,
                       double* cfl_dev, void* stream)
{
    int rc = claw2_validate(p);
    if (rc) return rc;
    if (!q_in || !q_out || !cfl_dev || (p->num_aux > 0 && !aux) || q_in == q_out) return CLAW2_ERR_INVALID;
    int nbx, nby;
    tiles(p, &nbx, &nby);
    if ((long long)nbx * (long long)nby > CLAW2_NOALLOC_MAX_TILES) return CLAW2_ERR_SIZE;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return CLAW2_ERR_CUDA;
    if (dev < 0 || dev >= kMaxDevices) return CLAW2_ERR_UNSUPPORTED;
    // Set-up, once per device, with that device current: the name of a
    // __device__ variable is only a host-side stand-in, so the kernel gets the
    // address the runtime reports for this device.
    void* scratch = g_noalloc_addr[dev].load(std::memory_order_acquire);
    if (!scratch) {
        if (cudaGetSymbolAddress(&scratch, g_noalloc_scratch) != cudaSuccess || !scratch) return CLAW2_ERR_CUDA;
        g_noalloc_addr[dev].store(scratch, std::memory_order_release);
    }
    // the array keeps the previous call's contents; the arrival counter must start at zero
    if (cudaMemsetAsync(scratch, 0, 64, S(stream)) != cudaSuccess) return CLAW2_ERR_CUDA;
    return claw2_step(p, q_in, q_out, aux, dt, scratch, cfl_dev, stream);
}

// ---------------------------------------------------------------------------
// host-buffer session
// ---------------------------------------------------------------------------
struct claw2_session {
    claw2_problem p;
    claw2_layout L;
    double *q0, *q1, *aux, *ref, *cfl;
    void* scratch;
    claw2_control* ctrl;       // device
    claw2_control* ctrl_host;  // pinned
    cudaStream_t stream;
};

int claw2_session_create(const claw2_problem* p, claw2_session** out)
{
    int rc = claw2_validate(p);
    if (rc) return rc;
    if (!out) return CLAW2_ERR_INVALID;
    claw2_session* s = new (std::nothrow) claw2_session;
    if (!s) return CLAW2_ERR_NOMEM;
    std::memset(s, 0, sizeof *s);
    s->p = *p;
    claw2_get_layout(p, &s->L);
    const size_t qb = sizeof(double) * s->L.q_elems;
    const size_t nref = (size_t)(p->num_eqn > p->num_aux ? p->num_eqn : p->num_aux) *
                        (p->mx + 2 * CLAW2_NUM_GHOST) * (p->my + 2 * CLAW2_NUM_GHOST);
    bool ok = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) == cudaSuccess;
    ok = ok && cudaMalloc(&s->q0, qb) == cudaSuccess && cudaMalloc(&s->q1, qb) == cudaSuccess;
    ok = ok && cudaMalloc(&s->ref, sizeof(double) * nref) == cudaSuccess;
    ok = ok && cudaMalloc(&s->cfl, sizeof(double)) == cudaSuccess;
    ok = ok && cudaMalloc(&s->scratch, claw2_scratch_bytes(p)) == cudaSuccess;
    ok = ok && cudaMalloc(&s->ctrl, sizeof(claw2_control)) == cudaSuccess;
    ok = ok && cudaMallocHost(&s->ctrl_host, sizeof(claw2_control)) == cudaSuccess;
    if (ok && p->num_aux > 0) ok = cudaMalloc(&s->aux, sizeof(double) * s->L.aux_elems) == cudaSuccess;
    ok = ok && cudaMemset(s->q0, 0, qb) == cudaSuccess && cudaMemset(s->q1, 0, qb) == cudaSuccess;
    ok = ok && cudaMemset(s->scratch, 0, claw2_scratch_bytes(p)) == cudaSuccess;
    if (!ok) { claw2_session_destroy(s); return CLAW2_ERR_NOMEM; }
    *out = s;
    return CLAW2_OK;
}

int claw2_session_destroy(claw2_session* s)
{
    if (!s) return CLAW2_OK;
    if (s->stream) cudaStreamSynchronize(s->stream);
    cudaFree(s->q0); cudaFree(s->q1); cudaFree(s->ref); cudaFree(s->cfl); cudaFree(s->scratch);
    cudaFree(s->ctrl); cudaFree(s->aux);
    if (s->ctrl_host) cudaFreeHost(s->ctrl_host);
    if (s->stream) cudaStreamDestroy(s->stream);
    delete s;
    return CLAW2_OK;
}

static int upload_aux(claw2_session* s, const double* aux, bool ghosts)
{
    const claw2_problem* p = &s->p;
    if (p->num_aux == 0) return CLAW2_OK;
    if (!aux) return CLAW2_ERR_INVALID;
    const size_t n = (size_t)p->num_aux * (p->mx + (ghosts ? 2 * CLAW2_NUM_GHOST : 0)) *
                     (p->my + (ghosts ? 2 * CLAW2_NUM_GHOST : 0));
    if (cudaMemcpyAsync(s->ref, aux, n * sizeof(double), cudaMemcpyHostToDevice, s->stream) != cudaSuccess)
        return CLAW2_ERR_CUDA;
    int rc = conv(p, p->num_aux, s->ref, s->aux, true, ghosts, s->stream);
    if (rc) return rc;
    if (!ghosts) return claw2_fill_aux_ghosts(p, s->aux, s->stream);
    return CLAW2_OK;
}

int claw2_session_step2(claw2_session* s, const double* qold, double* qnew, const double* aux, double dt,
                        double* cfl)
{
    if (!s || !qold || !qnew || !cfl) return CLAW2_ERR_INVALID;
    const claw2_problem* p = &s->p;
    const size_t n = (size_t)p->num_eqn * (p->mx + 2 * CLAW2_NUM_GHOST) * (p->my + 2 * CLAW2_NUM_GHOST);
    int rc;
    if ((rc = upload_aux(s, aux, true))) return rc;
    if (cudaMemcpyAsync(s->ref, qold, n * sizeof(double), cudaMemcpyHostToDevice, s->stream) != cudaSuccess)
        return CLAW2_ERR_CUDA;
    if ((rc = conv(p, p->num_eqn, s->ref, s->q0, true, true, s->stream))) return rc;
    bool chained = false;
    if ((rc = step_once(p, s->q0, s->q1, s->aux, dt, s->scratch, s->cfl, s->stream, true, &chained))) return rc;
    if ((rc = conv(p, p->num_eqn, s->q1, s->ref, false, true, s->stream, chained))) return rc;
    if (cudaMemcpyAsync(qnew, s->ref, n * sizeof(double), cudaMemcpyDeviceToHost, s->stream) != cudaSuccess)
        return CLAW2_ERR_CUDA;
    if (cudaMemcpyAsync(cfl, s->cfl, sizeof(double), cudaMemcpyDeviceToHost, s->stream) != cudaSuccess)
        return CLAW2_ERR_CUDA;
    if (cudaStreamSynchronize(s->stream) != cudaSuccess) return CLAW2_ERR_CUDA;
    return std::isnan(*cfl) ? CLAW2_ERR_NONFINITE : CLAW2_OK;
}

int claw2_session_evolve(claw2_session* s, double* q, const double* aux, double* t, double* dt, double tend,
                         double cfl_max, double cfl_desired, double dt_max, int64_t max_steps, double* status)
{
    if (!s || !q || !t || !dt) return CLAW2_ERR_INVALID;
    const claw2_problem* p = &s->p;
    const size_t n = (size_t)p->num_eqn * p->mx * p->my;
    int rc;
    if ((rc = upload_aux(s, aux, false))) return rc;
    if (cudaMemcpyAsync(s->ref, q, n * sizeof(double), cudaMemcpyHostToDevice, s->stream) != cudaSuccess)
        return CLAW2_ERR_CUDA;
    if ((rc = conv(p, p->num_eqn, s->ref, s->q0, true, false, s->stream))) return rc;
    if ((rc = claw2_fill_ghosts(p, s->q0, s->stream))) return rc;
    if ((rc = claw2_control_init(s->ctrl_host, *t, *dt, tend, cfl_max, cfl_desired, dt_max, 1, 0, max_steps, cfl_desired)))
        return rc;
    if (cudaMemcpyAsync(s->ctrl, s->ctrl_host, sizeof(claw2_control), cudaMemcpyHostToDevice, s->stream) != cudaSuccess)
        return CLAW2_ERR_CUDA;
    for (;;) {
        // the controller's own estimate of the steps left (to tend and to
        // max_steps), at most 256 per batch: the host reads the controller
        // only between batches, and steps launched after it is done return
        // at once
        const claw2_control* h = s->ctrl_host;
        double left = (double)(h->max_steps - h->iter);
        if (h->dt > 0.0) left = std::min(left, (h->tend - h->t) / h->dt + 1.0);
        const int batch = (int)std::max(1.0, std::min(256.0, left));
        if ((rc = claw2_advance(p, s->q0, s->q1, s->aux, s->ctrl, s->scratch, batch, s->stream))) return rc;
        if (cudaMemcpyAsync(s->ctrl_host, s->ctrl, sizeof(claw2_control), cudaMemcpyDeviceToHost, s->stream) != cudaSuccess)
            return CLAW2_ERR_CUDA;
        if (cudaStreamSynchronize(s->stream) != cudaSuccess) return CLAW2_ERR_CUDA;
        if (s->ctrl_host->done) break;
    }
    const claw2_control* c = s->ctrl_host;
    double* cur = c->cur ? s->q1 : s->q0;
    if ((rc = conv(p, p->num_eqn, cur, s->ref, false, false, s->stream))) return rc;
    if (cudaMemcpyAsync(q, s->ref, n * sizeof(double), cudaMemcpyDeviceToHost, s->stream) != cudaSuccess)
        return CLAW2_ERR_CUDA;
    if (cudaStreamSynchronize(s->stream) != cudaSuccess) return CLAW2_ERR_CUDA;
    *t = c->t;
    *dt = c->dt;
    if (status) {
        status[0] = c->status_cflmax; status[1] = c->status_dtmin; status[2] = c->status_dtmax;
        status[3] = (double)c->numsteps; status[4] = (double)c->rejected;
    }
    return c->error;
}

}  // extern "C"
