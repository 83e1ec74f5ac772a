"""A class byte without a rule (include/ebem.h, ebem_assemble_sa_selected): the
lag's block is zero, the others are those of their rules."""
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu


def test_class_without_rule():
    if not cuda_available():
        pytest.skip("no CUDA device")
    import torch
    import elastodynamicebem_b200.core as core
    from elastodynamicebem_b200 import mesh, problem
    prm = problem.ProblemParams(1, 1, 2, 1, 20)
    dm = core.DeviceMesh(mesh.screen_uniform(4))
    E = core.assemble_sa(dm, prm, 7)
    L, N = E.shape[0], dm.N
    cls = torch.zeros((N * N, L), dtype=torch.uint8, device="cuda")
    off = torch.rand((N, N, L), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda") < 0.3
    cls[off.view(N * N, L)] = 200
    out = torch.full((L, 3 * N, 3 * N), float("nan"), dtype=torch.float64, device="cuda")
    got, counts = core.assemble_sa_selected(dm, prm, cls, [(7, 1), (3, 1)], 0, L, out=out)
    gone = off.permute(2, 1, 0).repeat_interleave(3, 1).repeat_interleave(3, 2)        # [lag, source, field]
    want = torch.where(gone, torch.zeros_like(E), E)
    assert bool((want != E).any())
    assert torch.equal(got, want)
    assert counts[1] == 0
