"""Numerical post-processing where 8 lanes share an item and where the time sum
runs over (instant, triangle): rules of fewer nodes than lanes, of a number not
a multiple of 8, few and many (time, point) pairs, against the oracle."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sub,n_sing,npts,ntimes", [(1, 3, 1, 1), (1, 7, 1, 40), (4, 19, 1, 5), (16, 3, 33, 1), (1, 3, 40, 9),
                                                      (4, 3, 90, 40)])
def test_pp_num_lanes(oracle, n_sub, n_sing, npts, ntimes):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import torch
    import elastodynamicebem_b200.core as core
    from elastodynamicebem_b200 import mesh, problem
    m, prm = mesh.icosphere(1), problem.ProblemParams(1, 1, 1, 1, 40)
    rng = np.random.default_rng(11)
    phi = rng.normal(size=(prm.nT, 3 * m.numberTriangles))
    pts = rng.normal(size=(npts, 3)) * 0.2 + 1.1
    times = np.linspace(0.3, 1.0, ntimes)
    dm = core.DeviceMesh(m)
    for variant in (core.PP_POINT, core.PP_LAYER):
        u = core.pp_gpu(dm, prm, torch.tensor(phi, device="cuda"), pts, times, n_sub, n_sing, variant).cpu().numpy().transpose(2, 1, 0)
        uo = oracle.pp_gpu(m, prm, phi.T, pts, times, n_sub, n_sing, variant)
        # the same terms of at most 80 x 76 nodes x 40 instants in another order
        assert u.shape == uo.shape
        assert np.abs(u - uo).max() <= 1e-11 * np.abs(uo).max()
