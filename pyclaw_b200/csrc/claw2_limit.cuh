// claw2_limit.cuh -- the TVD limiters (philim.f90:18-55) of a ratio already formed.
#pragma once

#include <cuda_runtime.h>

namespace claw2 {

// philim (claw2_kernels.cuh) as a function of the ratio
__device__ __forceinline__ double philim_r(double r, int meth)
{
    double t, u;
    switch (meth) {
    case 2:
        t = 1.0 < 2.0 * r ? 1.0 : 2.0 * r;
        u = 2.0 < r ? 2.0 : r;
        t = t > u ? t : u;
        return 0.0 > t ? 0.0 : t;
    case 3:
        return (r + fabs(r)) / (1.0 + fabs(r));
    case 4: {
        const double c = (1.0 + r) / 2.0;
        t = c < 2.0 ? c : 2.0;
        t = t < 2.0 * r ? t : 2.0 * r;
        return 0.0 > t ? 0.0 : t;
    }
    case 5:
        return r;
    default:
        t = 1.0 < r ? 1.0 : r;
        return 0.0 > t ? 0.0 : t;
    }
}

// philim of a finite ratio for the limiters that are minima and maxima
__device__ __forceinline__ double positive_part(double t) { return __double2hiint(t) < 0 ? 0.0 : t; }
__device__ __forceinline__ double philim_mc(double r)
{
    const double c = (1.0 + r) * 0.5, r2 = r + r;
    const double t = c < 2.0 ? c : 2.0;
    return positive_part(t < r2 ? t : r2);
}
__device__ __forceinline__ double philim_minmod(double r) { return positive_part(1.0 < r ? 1.0 : r); }
__device__ __forceinline__ double philim_superbee(double r)
{
    const double r2 = r + r, t = 1.0 < r2 ? 1.0 : r2, u = 2.0 < r ? 2.0 : r;
    return positive_part(t > u ? t : u);
}

}  // namespace claw2
