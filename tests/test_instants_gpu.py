"""Instants t - k dt of several output times (post-processings): together as one
by one, whether the times lie on the time grid or not.

Each (time, point) sums the same terms in the same order either way: the
closed form bit for bit, the numerical one, which may split its nodes over
lanes, within 100 roundings (1e-14 of the largest value)."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu

NT, DT = 30, 1 / 30
TIMES = {
    "off": [0.013, 0.11, 0.345, 0.346, 0.7771, 0.99],
    "unordered": [0.99, 0.013, 0.7771, 0.11],
    "repeated": [0.5001, 0.2, 0.5001, 0.2],
    "one_phase": [0.01 + k * DT for k in (3, 1, 20, 7)],
    "grid": [k * DT for k in (1, 2, 3, 17, 29, 30)],
    "mixed": [10 * DT, 0.41, 11 * DT, 0.4100001, 0.0, -1.0],
    "one": [0.61],
    "none": [0.0, -0.5],
}


@pytest.mark.parametrize("name", list(TIMES))
def test_together(name):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import torch
    import elastodynamicebem_b200.core as core
    from elastodynamicebem_b200 import mesh, problem
    prm = problem.ProblemParams(1, 1, 1, 1, NT)
    dm = core.DeviceMesh(mesh.icosphere(1))
    rng = np.random.default_rng(1)
    phi = torch.from_numpy(rng.normal(size=(NT, 3 * dm.N))).cuda()
    pts = 1.3 * rng.normal(size=(3, 3))
    times = np.array(TIMES[name])
    for call, tol in ((lambda t: core.pp_sa(dm, prm, phi, pts, t), 0.0),
                      (lambda t: core.pp_gpu(dm, prm, phi, pts, t, 4, 3, core.PP_POINT), 1e-14)):
        got = call(times)
        want = torch.cat([call(times[q:q + 1]) for q in range(len(times))])
        assert got.shape == want.shape
        assert bool(want.any()) == (name != "none")
        assert float((got - want).abs().max()) <= tol * float(want.abs().max())
