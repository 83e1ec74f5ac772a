"""Marching on the banded blocks: step counts around the block of 8 steps of
the history product, fewer and more lags than steps, against the dense marching."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nT,steps", [(3, 20, 1), (3, 20, 7), (3, 20, 8), (4, 20, 9), (4, 20, 16), (5, 40, 39), (5, 6, 21)])
def test_banded_march_blocks(n, nT, steps):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import torch
    import elastodynamicebem_b200.core as core
    from elastodynamicebem_b200 import mesh, problem
    dm = core.DeviceMesh(mesh.screen_uniform(n))
    prm = problem.ProblemParams(1, 1, 2, 1, nT)
    b = torch.tensor(np.random.default_rng(5).normal(size=(steps, 3 * dm.N)), device="cuda")
    E = core.assemble_sa(dm, prm, 7, 0, core.num_blocks(dm, prm))
    phi = core.march(E, b).cpu().numpy()
    phib = core.BandedOperator(dm, prm, 7).march(b).cpu().numpy()
    # the same recurrence with sums in another order: the blocks agree to 1e-13,
    # the marching of up to 39 steps is stable, so a factor 10 a step block at most
    assert np.abs(phib - phi).max() <= 1e-11 * np.abs(phi).max()
