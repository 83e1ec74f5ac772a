"""Both precision modes of the semi-analytic assembly give the FP64 blocks
(include/ebem.h, EBEM_PREC_MIXED): bit for bit, whatever the output."""
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu


def test_modes_give_the_same_blocks():
    if not cuda_available():
        pytest.skip("no CUDA device")
    import torch
    import elastodynamicebem_b200.core as core
    from elastodynamicebem_b200 import mesh, problem
    prm = problem.ProblemParams(1, 1, 2, 1, 20)
    dm = core.DeviceMesh(mesh.screen_graded(6, 8, 2.0))
    E = core.assemble_sa(dm, prm, 7)
    L = E.shape[0]
    assert bool(E.any())
    assert torch.equal(core.assemble_sa(dm, prm, 7, prec=core.PREC_MIXED), E)
    assert torch.equal(core.BandedOperator(dm, prm, 7, prec=core.PREC_MIXED).to_dense(),
                       core.BandedOperator(dm, prm, 7).to_dense())
    cls = torch.randint(0, 2, (dm.N, dm.N, L), dtype=torch.uint8, device="cuda")
    rules = [(3, 1), (7, 1)]
    a, b = (core.assemble_sa_selected(dm, prm, cls, rules, 0, L, prec=p)[0] for p in (core.PREC_FP64, core.PREC_MIXED))
    assert bool(a.any()) and torch.equal(a, b)
