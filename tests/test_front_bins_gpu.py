"""Numerical-inner assemblies (E and K) by front arrivals: lag windows, rules beyond one
chunk of node pairs, more lags than one launch takes, and the kernel of few
node pairs, against the oracle's evaluation lag by lag."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu

# The entries are sums over at most 5776 node pairs of terms that the two
# evaluations order and split differently; each term is at most a few times the
# largest entry's, so the difference stays below 1e4 units of 2^-53 of that
# entry, about 1e-12.
TOL = 1e-12


@pytest.mark.parametrize("refine,rule,nT,lag0,nlag", [
    (1, (3, 1, 3), 40, 0, 41),           # 9 node pairs: partly filled warp
    (1, (7, 16, 3), 40, 5, 1),           # one lag
    (1, (7, 16, 3), 400, 100, 7),        # window that starts between the fronts
    (1, (12, 64, 7), 40, 3, 5),          # 42 inner nodes a chunk
    (1, (19, 16, 19), 40, 0, 4),         # 26 inner nodes a chunk, the last one short
    (0, (7, 4, 3), 1500, 300, 600),      # two launches
    (2, (3, 1, 1), 40, 0, 41),           # thread per pair
])
def test_ghc_front_bins(oracle, refine, rule, nT, lag0, nlag):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import elastodynamicebem_b200.core as core
    from elastodynamicebem_b200 import mesh, problem
    m = mesh.icosphere(refine)
    x = m.coordinates + np.random.default_rng(3).uniform(-0.02, 0.02, m.coordinates.shape) * m.lMin
    m = mesh.Mesh(x, m.triangles)        # no distance equal to a front's by symmetry
    prm = problem.ProblemParams(1, 1, 1, 1, nT)
    E = core.assemble_ghc(core.DeviceMesh(m), prm, *rule, lag0, nlag, sa_diagonal=False).cpu().numpy()
    Eo = oracle.assemble_ghc(m, prm, *rule, lag0, nlag)
    assert np.abs(Eo).max() > 0
    assert np.abs(E - Eo).max() <= TOL * np.abs(Eo).max()


@pytest.mark.parametrize("refine,rule,fix,T,nT,lag0,nlag", [
    (1, (3, 1, 1), False, 1, 20, 0, 6),            # 3 node pairs a triangle: one partly filled warp
    (1, (3, 64, 3), False, 1, 20, 0, 21),          # chunks of 73 inner nodes
    (1, (19, 4, 12), True, 1, 20, 0, 21),          # 26 inner nodes a chunk
    (1, (7, 4, 3), False, 1, 20, 2, 1),            # one lag, with the linear term
    (1, (12, 4, 3), True, 1, 100, 30, 9),          # window that starts between the fronts
    (0, (7, 4, 3), False, 0.4, 600, 0, 530),       # two launches
    (3, (3, 1, 1), False, 1, 20, 1, 4),            # thread per pair
])
def test_k_front_bins(oracle, refine, rule, fix, T, nT, lag0, nlag):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import elastodynamicebem_b200.core as core
    from elastodynamicebem_b200 import mesh, problem
    m = mesh.icosphere(refine)
    x = m.coordinates + np.random.default_rng(3).uniform(-0.02, 0.02, m.coordinates.shape) * m.lMin
    m = mesh.Mesh(x, m.triangles)
    prm = problem.ProblemParams(1, 1, 1, T, nT)
    dm = core.DeviceMesh(m)
    LK = core.num_blocks_dir(dm, prm)[1]
    K = core.assemble_k(dm, prm, *rule, 0, lag0, nlag, fix=fix).cpu().numpy()
    Ko = oracle.assemble_k(m, prm, *rule, lag0, nlag, nblocks=LK, fix=fix)
    # the oracle's third differences of levels that grow like (t / dt)^3
    tol = TOL + 1e-15 * (lag0 + nlag) ** 3
    assert np.abs(Ko).max() > 0
    assert np.abs(K - Ko).max() <= tol * np.abs(Ko).max()
