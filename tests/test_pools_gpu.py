"""A device whose free memory lies in the pool of destroyed handles' storage:
a call's workspace gets it.

A child process preloads a shim that refuses large allocations from any pool
until another pool has been trimmed, as a full device would."""
import os
import shutil
import subprocess
import sys

import pytest

from conftest import ROOT, cuda_available

pytestmark = pytest.mark.gpu

SHIM = r"""
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <cstdlib>

static cudaMemPool_t held = nullptr;      // the pool that holds the rest of the device
static bool trimmed = false;
extern "C" cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t s) {
    using F = cudaError_t (*)(void**, size_t, cudaMemPool_t, cudaStream_t);
    if (!held) held = pool;               // the first allocation is a handle's
    if (pool != held && n > 4000000 && !trimmed) return cudaErrorMemoryAllocation;
    return ((F)dlsym(RTLD_NEXT, "cudaMallocFromPoolAsync"))(p, n, pool, s);
}
extern "C" cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t n) {
    using F = cudaError_t (*)(cudaMemPool_t, size_t);
    if (pool == held && n == 0) trimmed = true;
    return ((F)dlsym(RTLD_NEXT, "cudaMemPoolTrimTo"))(pool, n);
}
"""

# the node table comes from the storage pool, the 4.6 MB of blocks from the other one
CODE = """
import sys; sys.path.insert(0, sys.argv[1])
from elastodynamicebem_b200 import core, mesh, problem
prm = problem.ProblemParams(1, 1, 1, 1, 10)
dm = core.DeviceMesh(mesh.icosphere(1))
core.rhs(dm, prm, 7, problem.DATUM_RADIAL_SIN)
phi, _ = core.timemarch_sa(dm, prm, 7, problem.DATUM_RADIAL_SIN)
assert bool(phi.isfinite().all()) and bool(phi.any())
print("done")
"""


def test_memory_held_by_the_other_pool(tmp_path):
    if not cuda_available():
        pytest.skip("no CUDA device")
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    (tmp_path / "shim.cpp").write_text(SHIM)
    so = str(tmp_path / "shim.so")
    subprocess.run([gxx, "-O1", "-fPIC", "-shared", "-I", "/usr/local/cuda/include", str(tmp_path / "shim.cpp"), "-o", so,
                    "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", CODE, ROOT], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=so))
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr
