"""An infinity or NaN in the blocks of one lag reaches the steps from that lag
on and no step before (the history of 8 steps is one product, in which the
first steps do not use its last lags)."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu

L, NT = 16, 27


def _check(march, blocks, lag, value):
    """march(blocks) with one entry of blocks[lag] not finite, against that lag's zeros up to step lag - 1."""
    clean, bad = blocks.clone(), blocks.clone()
    clean[lag] = 0
    bad[lag, 5, 7] = value
    want, got = march(clean), march(bad)
    assert bool(got[:lag].isfinite().all())
    assert float((got[:lag] - want[:lag]).abs().max()) <= 1e-12 * float(want[:lag].abs().max())
    assert not bool(got[lag].isfinite().all())


# lags used first in the first block, in the middle and at the end of a later one, and at a block's first step
@pytest.mark.parametrize("lag", [3, 8, 12, 15])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("n3", [96, 129])
def test_march(n3, lag, value):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import torch
    import elastodynamicebem_b200.core as core
    g = torch.Generator(device="cuda").manual_seed(1)
    E = 0.1 / n3 * torch.randn((L, n3, n3), generator=g, dtype=torch.float64, device="cuda")
    E[0] += torch.eye(n3, dtype=torch.float64, device="cuda")
    b = torch.randn((NT, n3), generator=g, dtype=torch.float64, device="cuda")
    _check(lambda M: core.march(M, b), E, lag, value)


@pytest.mark.parametrize("lag", [3, 12])
def test_march_dn(lag):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import torch
    import elastodynamicebem_b200.core as core
    from elastodynamicebem_b200 import mesh, problem
    m = mesh.prism_bar(1.0, 1.0, 3.0, 0.5)
    prm = problem.ProblemParams(1, 1, 2, 1, NT)
    dm = core.DeviceMesh(m)
    R, C = 3 * m.numberTriangles, 3 * m.number_nodes
    g = torch.Generator(device="cuda").manual_seed(2)
    K = 1e-3 / C * torch.randn((L, R, C), generator=g, dtype=torch.float64, device="cuda")
    inc = torch.from_numpy(np.kron(m.vertex_triangle_incidence().T * (m.area / 6)[:, None], np.eye(3))).cuda()
    K[0] += 0.25 * inc
    V = torch.eye(R, dtype=torch.float64, device="cuda")[None]
    gV = torch.randn((NT, R), generator=g, dtype=torch.float64, device="cuda")
    _check(lambda M: core.march_dn(dm, prm, V, M, gV), K, lag, float("nan"))
