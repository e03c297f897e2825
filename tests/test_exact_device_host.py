"""recip_rn, sqrt_rn, quot_rn and low_quot of claw2_exact.cuh, compiled for the host:
the bits of the IEEE operations on operands next to midpoints, whatever the error
of the hardware's approximations that they start from."""
import ctypes

import numpy as np
import pytest

from exact_operands import cases
from host_device import compile_host

SOURCE = r"""
#include <cuda_runtime.h>
#include "claw2_exact.cuh"
using namespace claw2;
extern "C" void run(int op, long n, const double* x, const double* y, double* out, double seed_error)
{
    emu::seed_error = seed_error;
    for (long i = 0; i < n; i++)
        out[i] = op == 0 ? recip_rn(y[i]) : op == 1 ? sqrt_rn(x[i]) : op == 2 ? quot_rn(x[i], y[i], recip_rn(y[i]))
                                                                             : low_quot(x[i], y[i], recip_rn(y[i]));
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    lib = ctypes.CDLL(compile_host(SOURCE, tmp_path_factory.mktemp("exact")))
    lib.run.argtypes = [ctypes.c_int, ctypes.c_long] + 3 * [ctypes.c_void_p] + [ctypes.c_double]
    lib.run.restype = None
    return lib


# relative errors of the seed on top of the truncation to 20 bits
@pytest.mark.parametrize("seed_error", [0.0, 2.0 ** -21, 2.0 ** -20, -2.0 ** -22, -2.0 ** -20])
def test_bits_of_the_ieee_operations(lib, seed_error):
    for op, x, y, want in cases(1):
        got = np.empty_like(want)
        lib.run(op, x.size, x.ctypes.data, y.ctypes.data, got.ctypes.data, seed_error)
        wrong = np.flatnonzero(got != want)
        assert wrong.size == 0, (op, wrong.size, x[wrong[0]].hex(), y[wrong[0]].hex(), got[wrong[0]].hex())
