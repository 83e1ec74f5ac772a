"""Windows of few lags of the numerical assemblies (E and K), which take another
kernel than the whole range where they have few node pairs, skip the pairs that
no front reaches and evaluate the constants of earlier arrivals apart: equal to
the lags of the whole assembly.

Both sum at most 2016 node pairs in another order: 1e4 units of 2^-53 of the
largest entry, 1e-12; K's thread kernel forms third differences of levels that
grow like (t / dt)^3 (1e-15 per unit of it)."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu

WINDOWS = [(0, 1), (0, 4), (1, 1), (2, 2), (3, 1), (20, 1), (20, 4), (20, 12), (37, 3)]


@pytest.fixture(scope="module")
def setup():
    if not cuda_available():
        pytest.skip("no CUDA device")
    import elastodynamicebem_b200.core as core
    from elastodynamicebem_b200 import mesh, problem
    m = mesh.prism_bar(1.0, 1.0, 3.0, 1 / 3)                     # 252 triangles: enough pairs for the thread kernels
    x = m.coordinates + np.random.default_rng(3).uniform(-0.02, 0.02, m.coordinates.shape) * m.lMin
    m = mesh.Mesh(x, m.triangles)
    return core, core.DeviceMesh(m), problem.ProblemParams(1, 1, 2, 1, 40)


@pytest.mark.parametrize("rule", [(3, 1, 1), (3, 1, 3), (7, 1, 3), (3, 4, 3), (7, 4, 3)])
def test_ghc(setup, rule):
    core, dm, prm = setup
    E = core.assemble_ghc(dm, prm, *rule, 0, 40, sa_diagonal=False)
    for lag0, n in WINDOWS:
        W = core.assemble_ghc(dm, prm, *rule, lag0, n, sa_diagonal=False)
        assert float((W - E[lag0:lag0 + n]).abs().max()) <= 1e-12 * float(E.abs().max()), (lag0, n)


@pytest.mark.parametrize("fix", [False, True])
@pytest.mark.parametrize("rule", [(3, 1, 1), (3, 1, 3), (7, 1, 3), (3, 4, 3)])
def test_k(setup, rule, fix):
    core, dm, prm = setup
    K = core.assemble_k(dm, prm, *rule, 16, 0, 40, fix=fix)
    for lag0, n in WINDOWS:
        W = core.assemble_k(dm, prm, *rule, 16, lag0, n, fix=fix)
        tol = 1e-12 + 1e-15 * (lag0 + n) ** 3
        assert float((W - K[lag0:lag0 + n]).abs().max()) <= tol * float(K.abs().max()), (lag0, n)
