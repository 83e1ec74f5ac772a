"""The inverse of an assembled E_0 (csrc/inverse.cu): entries of many sizes on
edge-graded screens, condition numbers up to some 1e6.

Tolerance: the solution by an inverse with partial pivoting errs by at most
about n * 2.2e-16 * condition in the norm (the rounding of b = A x included);
the pivoting of a wrong row shows as an error of order 1."""
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb,beta", [(6, 6, 2.0), (8, 16, 3.0), (12, 20, 2.0)])
def test_graded_screen(na, nb, beta):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import torch
    import elastodynamicebem_b200.core as core
    from elastodynamicebem_b200 import mesh, problem
    m = mesh.screen_graded(na, nb, beta)
    prm = problem.ProblemParams(1, 1, 2, 1, 40)
    A = core.assemble_sa(core.DeviceMesh(m), prm, 7, 0, 1)[0].contiguous()
    n = A.shape[0]
    cond = float(torch.linalg.cond(A))
    assert n * 2.2e-16 * cond < 1e-3
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn((3, n), generator=g, dtype=torch.float64, device="cuda")
    lu = core.DeviceLU(A)
    got = lu.solve((x @ A.T).contiguous())
    lu.close()
    assert float((got - x).norm() / x.norm()) <= n * 2.2e-16 * cond
