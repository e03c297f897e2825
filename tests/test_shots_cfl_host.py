"""The CFL numbers of the multi-shot step, as its CTAs collect them (collect_cfl of
claw2_kernels.cuh over the shots' counters and cells, which lie next to one
another): whatever the order in which the CTAs of all shots arrive, every shot
reports its own maximum, and counters and cells are zero for the next step."""
import ctypes

import numpy as np
import pytest

from host_device import compile_host

SOURCE = r"""
#include <cuda_runtime.h>
#include "../../include/claw2.h"
#include "claw2_kernels.cuh"
using namespace claw2;

// arrivals: (shot, CFL number or NaN for a state that is not finite), in order; the
// arguments as shots_step_kernel has them
extern "C" void arrive(int n, const int* shot, const double* cfl, int ntiles, unsigned* tickets, double* cells, double* out)
{
    DevCtx ctx{nullptr};
    for (int k = 0; k < n; k++) {
        StepArgs a;
        std::memset(&a, 0, sizeof a);
        a.ticket = tickets + shot[k];
        a.partials = cells + shot[k];
        a.cfl_out = out + shot[k];
        collect_cfl(a, ctx, ntiles, cfl[k] == cfl[k] ? cfl[k] : 0.0, cfl[k] != cfl[k], false);
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    lib = ctypes.CDLL(compile_host(SOURCE, tmp_path_factory.mktemp("shots")))
    lib.arrive.restype = None
    return lib


@pytest.mark.parametrize("shots", [1, 4, 5, 12, 61, 64, 130])
def test_every_shot_reports_its_own_cfl(lib, shots):
    rng = np.random.default_rng(shots)
    counters = (shots * 4 + 255) // 256 * 64                    # claw2_shots_step's rounding
    scratch = np.zeros(counters + 2 * shots, dtype=np.uint32)
    tickets, cells = scratch.ctypes.data, scratch.ctypes.data + 4 * counters
    ntiles = 7
    for step in range(5):
        order = rng.permutation(np.repeat(np.arange(shots, dtype=np.int32), ntiles)).astype(np.int32)
        cfl = rng.random(order.size)
        bad = int(rng.integers(shots)) if step == 3 else -1
        if bad >= 0:
            cfl[np.flatnonzero(order == bad)[2]] = np.nan
        out = np.full(shots, -7.0)
        lib.arrive(order.size, ctypes.c_void_p(order.ctypes.data), ctypes.c_void_p(cfl.ctypes.data), ntiles,
                   ctypes.c_void_p(tickets), ctypes.c_void_p(cells), ctypes.c_void_p(out.ctypes.data))
        want = np.array([np.nan if s == bad else cfl[order == s].max() for s in range(shots)])
        assert np.array_equal(out, want, equal_nan=True), step
        assert not scratch.any(), step
