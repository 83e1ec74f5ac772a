"""The Gauss-Jordan inverse behind the marching's E_0 solve (csrc/inverse.cu)
at the edges of its panels (64 columns), its clusters' blocks (256 rows) and
update tiles (128 x 64), and past the largest matrix it takes.

Tolerance: random entries plus sqrt(n) on the diagonal give a condition number
of a few tens; an inverse by elimination with partial pivoting errs by a small
multiple of n * 2.2e-16 * condition, 2e-11 at n = 4097 with a factor of 10.
A permuted matrix (no large diagonal) makes every pivot leave its place."""
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu
TOL = 2e-11


@pytest.fixture(scope="module")
def ebem():
    if not cuda_available():
        pytest.skip("no CUDA device")
    import elastodynamicebem_b200.core as core
    return core


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 129, 255, 256, 257, 576, 2049, 4096, 4097])
def test_inverse(ebem, n):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.rand((n, n), generator=g, dtype=torch.float64, device="cuda") - 0.5
    A += n ** 0.5 * torch.eye(n, dtype=torch.float64, device="cuda")
    A = A[torch.randperm(n, generator=g, device="cuda")]
    b = torch.rand((3, n), generator=g, dtype=torch.float64, device="cuda")
    lu = ebem.DeviceLU(A)
    x = lu.solve(b.clone())
    lu.close()
    ref = torch.linalg.solve(A, b.T).T
    assert float((x - ref).norm() / ref.norm()) <= TOL


@pytest.mark.parametrize("n,column", [(40, 0), (300, 70), (300, 299)])
def test_zero_pivot(ebem, n, column):
    import torch
    from elastodynamicebem_b200.lib import EbemError
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.rand((n, n), generator=g, dtype=torch.float64, device="cuda")
    A[:, column] = 0.0
    with pytest.raises(EbemError) as e:
        ebem.DeviceLU(A)
    assert f"zero pivot {column + 1}" in str(e.value)
