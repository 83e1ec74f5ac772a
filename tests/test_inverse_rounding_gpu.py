"""Rounding of the inverse behind the marching (csrc/inverse.cu) on a matrix
with a diagonal of size 1 beside small entries, as E_0 has it.

An entry of size 1 that is rounded n times on its way ends some sqrt(n) / 2
units of 2^-53 off (20 at n = 1500); rounded once per panel of 64 columns, some
sqrt(n / 64) / 2 = 2.4.  With the product's own few units: 8 units in the norm.
The solution is refined in long double."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [500, 1500])
def test_diagonal(n):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import torch
    import elastodynamicebem_b200.core as core
    rng = np.random.default_rng(n)
    A = 0.1 / n ** 0.5 * rng.standard_normal((n, n)) + np.eye(n)
    b = rng.standard_normal(n)
    x, inv, Al, bl = np.zeros(n, np.longdouble), np.linalg.inv(A), A.astype(np.longdouble), b.astype(np.longdouble)
    for _ in range(4):
        x = x + inv @ (bl - Al.dot(x)).astype(np.float64)
    lu = core.DeviceLU(torch.from_numpy(A).cuda())
    got = lu.solve(torch.from_numpy(b).cuda()).cpu().numpy()
    lu.close()
    d = got - x
    assert float(np.sqrt((d ** 2).sum() / (x ** 2).sum())) <= 8 * 2.0 ** -53
