// claw2_launch.cuh -- launching step kernels, plain or chained.
#pragma once

#include <cuda_runtime.h>

#include "../../include/claw2.h"
#include "claw2_kernels.cuh"

namespace claw2 {

// Chained steps (launch_step with chained set): once every CTA of this step
// has started, the next step's CTAs may start on the SMs this step frees;
// each waits here until the step before it has completed and its writes are
// visible.  In a kernel launched without the attribute both instructions
// return at once.
__device__ __forceinline__ void chain_wait()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Launch kern, as a programmatic dependent of the previous kernel in the
// stream when chained is set (the kernel calls chain_wait before it reads
// anything).
template <class... KArgs, class... Args>
int launch_kernel(void (*kern)(KArgs...), dim3 grid, int threads, int smem, cudaStream_t st, bool chained,
                  Args... args)
{
    if (!chained) {
        kern<<<grid, threads, smem, st>>>(args...);
        return cudaGetLastError() == cudaSuccess ? CLAW2_OK : CLAW2_ERR_CUDA;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, args...) == cudaSuccess ? CLAW2_OK : CLAW2_ERR_CUDA;
}

// The unsplit acoustics step (claw2_march.cuh, claw2_acoustics.cu): rows of a
// CTA's tile when `cols` strips of my rows are stepped together, and the launch.
int march_rows_per_cta(int rp, long long cols, int my);
int launch_march(int rp, const StepArgs& a, cudaStream_t st, bool chained);

// The split acoustics step (claw2_rows.cuh, claw2_acoustics.cu).
int launch_rows(int rp, const StepArgs& a, cudaStream_t st, bool chained);

// The step of the Euler and shallow-water solvers (claw2_lean.cuh,
// claw2_lean.cu); the state buffers start on 16-byte boundaries.
constexpr int LEAN_T = 28;             // edge of its large tiles
int launch_lean(int rp, bool split, const StepArgs& a, cudaStream_t st, bool chained);

// The unsplit step of the p-system with f-waves and no capacity (claw2_psystem.cuh,
// claw2_psystem.cu).
int launch_psystem(const StepArgs& a, cudaStream_t st, bool chained);

}  // namespace claw2
