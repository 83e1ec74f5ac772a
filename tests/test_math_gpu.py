"""Device branches of csrc/sa_math.cuh (hardware seeds, exponent split) against
the host's long double functions over the ranges of their arguments.

Tolerances in units of 2^-52 of the result.  Reciprocal and square root: the
seed takes the upper 32 bits of its argument (relative error some 2^-19), the
correction leaves its cube (2^-56) and the rounding of the last operation
(2^-53): 1.  Logarithm and arctangent: as on the host (tests/test_front_cpu.py),
some eight roundings, two of them of the full result: 4."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT, cuda_available

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdint>
#include <cstring>
#include "sa_math.cuh"
using namespace ebem;
__global__ void k(int n, const double* x, const double* y, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = q_rcp(x[i]);
    out[n + i] = q_sqrt(x[i]);
    out[2 * n + i] = q_log(x[i]);
    out[3 * n + i] = q_atan2(y[i], x[i]);
}
extern "C" int device_math(int n, const double* x, const double* y, double* out) {
    double* d = nullptr;
    const size_t b = n * sizeof(double);
    cudaError_t e = cudaMalloc(&d, 6 * b);
    if (e != cudaSuccess) return (int)e;
    e = cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, y, b, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k<<<(n + 127) / 128, 128>>>(n, d, d + n, d + 2 * n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * n, 4 * b, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
"""


@pytest.fixture(scope="module")
def device_math(tmp_path_factory):
    if not cuda_available():
        pytest.skip("no CUDA device")
    from elastodynamicebem_b200 import build
    if not shutil.which(build.nvcc()):
        pytest.skip("nvcc not available")
    d = tmp_path_factory.mktemp("math")
    (d / "m.cu").write_text(SOURCE)
    so = str(d / "m.so")
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-I", os.path.join(ROOT, "elastodynamicebem_b200", "csrc"),
                    "-shared", str(d / "m.cu"), "-o", so], check=True)
    lib = C.CDLL(so)

    def run(x, y):
        out = np.empty((4, len(x)))
        ptr = lambda a: a.ctypes.data_as(C.c_void_p)
        assert lib.device_math(len(x), ptr(x), ptr(y), ptr(out)) == 0
        return out

    return run


def test_device_functions(device_math):
    rng = np.random.default_rng(3)
    x = np.concatenate([10.0 ** rng.uniform(-60, 60, 20000), 10.0 ** rng.uniform(-12, 12, 20000),
                        1 + rng.uniform(-0.4, 0.6, 20000), np.sqrt(0.5) * (1 + np.array([-2e-16, 0, 2e-16])),
                        2.0 ** np.arange(-40, 41), 2.0 ** np.arange(-40, 41) * (2 - 2.0 ** -51)])
    y = x * 10.0 ** rng.uniform(-10, 10, len(x))
    for k, edge in enumerate((1 / 8, 3 / 8)):          # the arctangent's breakpoints
        q = slice(20000 + 1000 * k, 21000 + 1000 * k)
        y[q] = x[q] * np.tan(np.pi * edge) * (1 + rng.uniform(-1e-15, 1e-15, 1000))
    got = device_math(x, y)
    xl, yl = x.astype(np.longdouble), y.astype(np.longdouble)
    eps = np.finfo(float).eps
    for g, want, units in zip(got, (1 / xl, np.sqrt(xl), np.log(xl), np.arctan2(yl, xl)), (1, 1, 4, 4)):
        assert np.all(np.abs(g - want) <= units * eps * np.abs(want))


def test_device_edges(device_math):
    x, y = np.array([0.0, -1.0, 0.0, 1.0, 1.0]), np.array([1.0, 1.0, 3.0, 0.0, 1.0])
    got = device_math(x, y)
    assert np.all(got[1, :3] == 0)                     # sqrt: 0 for x <= 0
    assert got[2, 3] == 0                              # log 1
    eps = np.finfo(float).eps
    want = np.array([np.pi / 2, np.pi / 2, np.pi / 2, 0, np.pi / 4])
    q = [0, 2, 3, 4]
    assert np.all(np.abs(got[3, q] - want[q]) <= eps)
