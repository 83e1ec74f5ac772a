"""Handles destroyed while a kernel that reads their storage is still queued:
the storage comes from a memory pool, whose frees wait for nothing, so destroying
the handle has to wait (include/ebem.h: calls with device outputs are
asynchronous on their stream)."""
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu

# Cycles that the first stream is kept busy with, some 0.1 s: the destruction and
# the next handle on a second stream take a few milliseconds.
BUSY = 200_000_000


def _problem(n):
    from elastodynamicebem_b200 import mesh, problem
    return mesh.screen_uniform(n), problem.ProblemParams(1, 1, 2, 1, 20)


def test_banded_destroyed_behind_to_dense():
    if not cuda_available():
        pytest.skip("no CUDA device")
    import torch
    import elastodynamicebem_b200.core as core
    m, prm = _problem(6)
    dm = core.DeviceMesh(m)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    op = core.BandedOperator(dm, prm, 7)
    want = op.to_dense()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(BUSY)
        got = op.to_dense(stream=a)
    op.close()
    assert a.query()                       # nothing of the operator's is queued any more
    # another operator of the same size, with other blocks, takes the storage
    with torch.cuda.stream(b):
        other = core.BandedOperator(dm, type(prm)(1, 1, 2, 1.3, 20), 3, stream=b)
    torch.cuda.synchronize()
    other.close()
    assert bool((got == want).all())


def test_mesh_destroyed_behind_assembly():
    if not cuda_available():
        pytest.skip("no CUDA device")
    import torch
    import elastodynamicebem_b200.core as core
    m, prm = _problem(6)
    dm = core.DeviceMesh(m)
    want = core.assemble_sa(dm, prm, 7)
    out = torch.empty_like(want).transpose(1, 2).contiguous()
    a = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(BUSY)
        got = core.assemble_sa(dm, prm, 7, 0, out.shape[0], out=out, stream=a)
    dm.close()
    assert a.query()
    other = core.DeviceMesh(_problem(7)[0])
    core.assemble_sa(other, prm, 12)
    torch.cuda.synchronize()
    assert bool((got == want).all())
