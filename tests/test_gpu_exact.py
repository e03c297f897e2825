"""recip_rn, sqrt_rn, quot_rn and low_quot of claw2_exact.cuh on the GPU: the bits of
the IEEE operations on operands next to midpoints, from the hardware's own
approximations.  A kernel of the test's own, compiled here, a thread per operand."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import gpu_helpers as H
from exact_operands import cases
from host_device import CSRC
from pyclaw_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cuda_runtime.h>
#include "claw2_exact.cuh"
using namespace claw2;
__global__ void kernel(int op, long n, const double* x, const double* y, double* out, double* plain)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        out[i] = op == 0 ? recip_rn(y[i]) : op == 1 ? sqrt_rn(x[i]) : op == 2 ? quot_rn(x[i], y[i], recip_rn(y[i]))
                                                                             : low_quot(x[i], y[i], recip_rn(y[i]));
        plain[i] = op == 0 ? 1.0 / y[i] : op == 1 ? sqrt(x[i]) : x[i] / y[i];
    }
}
extern "C" __attribute__((visibility("default"))) int run(int op, long n, const double* x, const double* y, double* out, double* plain, void* stream)
{
    kernel<<<256, 256, 0, (cudaStream_t)stream>>>(op, n, x, y, out, plain);
    return cudaGetLastError() != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact")
    (d / "exact.cu").write_text(SOURCE)
    out = str(d / "exact.so")
    subprocess.run([build.nvcc_path()] + build.NVCC_FLAGS + ["-I", CSRC, "-shared", "-cudart", "shared", "-o", out,
                                                             os.path.join(str(d), "exact.cu")], check=True)
    lib = ctypes.CDLL(out)
    lib.run.argtypes = [ctypes.c_int, ctypes.c_long] + 5 * [ctypes.c_void_p]
    return lib


@pytest.mark.parametrize("seed", [1, 2])
def test_bits_of_the_ieee_operations(lib, seed):
    t = H.torch()
    for op, x, y, want in cases(seed):
        dx, dy = t.from_numpy(np.ascontiguousarray(x)).cuda(), t.from_numpy(np.ascontiguousarray(y)).cuda()
        out, plain = t.empty_like(dx), t.empty_like(dx)
        assert lib.run(op, dx.numel(), dx.data_ptr(), dy.data_ptr(), out.data_ptr(), plain.data_ptr(), H.stream()) == 0
        got, cuda = out.cpu().numpy(), plain.cpu().numpy()
        assert np.array_equal(cuda, want), op
        wrong = np.flatnonzero(got != want)
        assert wrong.size == 0, (op, wrong.size, x[wrong[0]].hex(), y[wrong[0]].hex(), got[wrong[0]].hex())
