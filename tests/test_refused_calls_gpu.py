"""Calls of the CUDA runtime that are refused: the library takes its other path.

A child process preloads a shim that answers for the runtime as a device would
that cannot place a cluster, or that has no room for a large workspace; no such
launch or allocation is made."""
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

static unsigned cluster_of(const cudaLaunchConfig_t* c) {
    for (unsigned k = 0; k < c->numAttrs; k++)
        if (c->attrs[k].id == cudaLaunchAttributeClusterDimension) return c->attrs[k].val.clusterDim.x;
    return 1;
}
static unsigned most_clusters() {
    const char* v = std::getenv("SHIM_CLUSTER");
    return v ? (unsigned)std::atoi(v) : 1u << 30;
}
extern "C" cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
    if (cluster_of(c) > most_clusters()) {
        *n = 0;
        return cudaSuccess;
    }
    using F = cudaError_t (*)(int*, const void*, const cudaLaunchConfig_t*);
    return ((F)dlsym(RTLD_NEXT, "cudaOccupancyMaxActiveClusters"))(n, f, c);
}
extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) {
    if (cluster_of(c) > most_clusters()) return cudaErrorLaunchOutOfResources;
    using F = cudaError_t (*)(const cudaLaunchConfig_t*, const void*, void**);
    return ((F)dlsym(RTLD_NEXT, "cudaLaunchKernelExC"))(c, f, a);
}
extern "C" cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t s) {
    const char* v = std::getenv("SHIM_BYTES");
    if (v && n > (size_t)std::atoll(v)) return cudaErrorMemoryAllocation;
    using F = cudaError_t (*)(void**, size_t, cudaMemPool_t, cudaStream_t);
    return ((F)dlsym(RTLD_NEXT, "cudaMallocFromPoolAsync"))(p, n, pool, s);
}
"""


@pytest.fixture(scope="module")
def run_child(tmp_path_factory):
    if not cuda_available():
        pytest.skip("no CUDA device")
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("shim")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run([gxx, "-O1", "-fPIC", "-shared", "-I", "/usr/local/cuda/include", str(d / "shim.cpp"), "-o", so, "-ldl"],
                   check=True)

    def run(code, *args, **env):
        r = subprocess.run([sys.executable, "-c", "import sys; sys.path.insert(0, sys.argv[1])\n" + code, ROOT, *args],
                           capture_output=True, text=True, timeout=300,
                           env=dict(os.environ, LD_PRELOAD=so, **{k: str(v) for k, v in env.items()}))
        assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr

    return run


INVERSE = """
import torch
from elastodynamicebem_b200 import core
n = {n}
g = torch.Generator(device="cuda").manual_seed(n)
A = torch.rand((n, n), generator=g, dtype=torch.float64, device="cuda") - 0.5
A += n ** 0.5 * torch.eye(n, dtype=torch.float64, device="cuda")
b = torch.rand((2, n), generator=g, dtype=torch.float64, device="cuda")
ref = torch.linalg.solve(A, b.T).T
for x in (core.DeviceLU(A).solve(b.clone()), core.march(A[None], b)):
    assert float((x - ref).norm() / ref.norm()) <= 2e-11
A[:, n // 2] = 0
try:
    core.DeviceLU(A)
except core._lib.EbemError as e:
    assert "zero pivot %d" % (n // 2 + 1) in str(e), e
else:
    raise AssertionError("a singular matrix was inverted")
print("done")
"""


# (blocks a cluster may have, n): the panel of n rows asks for 2, 9 and 16 blocks of 256
@pytest.mark.parametrize("most,n", [(1, 300), (8, 2100), (8, 4096)])
def test_inverse_without_its_cluster(run_child, most, n):
    run_child(INVERSE.format(n=n), SHIM_CLUSTER=most)


def test_inverse_without_its_buffers(run_child):
    run_child(INVERSE.format(n=1000), SHIM_BYTES=12_000_000)         # two buffers of 8 MB in one


CALL = """
import numpy as np, torch
from elastodynamicebem_b200 import core, mesh, problem
prm = problem.ProblemParams(1, 1, 1, 1, 40)
dm = core.DeviceMesh(mesh.icosphere(2))
rng = np.random.default_rng(1)
phi = torch.from_numpy(rng.normal(size=(prm.nT, 3 * dm.N))).cuda()
pts = 1.5 * rng.normal(size=(50, 3))
torch.save({call}.contiguous(), sys.argv[2])
print("done")
"""


# 320 triangles: records of a field column 0.6 MB, M of a point 0.6 MB at 40 instants; off the grid each
# time has instants of its own, some 12 MB a point at 40 times
@pytest.mark.parametrize("call,limit", [
    ("core.assemble_sa(dm, prm, 7)", 8_000_000),
    ("core.assemble_sa(dm, prm, 7)", 700_000),
    ("core.pp_sa(dm, prm, phi, pts, prm.dt * np.arange(1, 41))", 4_000_000),
    ("core.pp_sa(dm, prm, phi, pts, np.linspace(0.013, 0.99, 40))", 2_000_000),
], ids=["sa", "sa_one_column", "pp_points", "pp_times"])
def test_workspace_that_does_not_fit(run_child, tmp_path, call, limit):
    """The same blocks, bit for bit, with workspaces above the limit refused; the
    post-processing sums its 1e4 terms in another order for fewer points or times
    a launch (1e4 units of 2^-53, 1e-12)."""
    import torch
    out = [str(tmp_path / f"{k}.pt") for k in range(2)]
    run_child(CALL.format(call=call), out[0])
    run_child(CALL.format(call=call), out[1], SHIM_BYTES=limit)
    a, b = (torch.load(o) for o in out)
    tol = 0.0 if "assemble" in call else 1e-12
    assert bool(a.any()) and float((a - b).abs().max()) <= tol * float(a.abs().max())
