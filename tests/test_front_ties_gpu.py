"""Fronts that reach a node pair exactly at a time level: t_k - r / c is zero as
the reference's formula rounds it (the product k dt, the quotient, their
difference), and the pair counts from the next level on.  With the product not
rounded (a fused multiply-add) the difference is the product's rounding error
and the pair would count one level earlier.

Two parallel triangles half a unit apart: their nodes of equal barycentric
coordinates lie at distance 0.5 exactly (x and y are computed alike, z is an
exact product).  With c_P = 2, c_S = 1 and dt = fl(1/20) the fronts meet them at
k = 5 and 10, where k dt rounds down to 0.25 and 0.5.  A front's jump is of the
size of the entry; without ties device and oracle differ by some 1e-13."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu

TOL = 1e-9
H = 0.125


def _pairs(n):
    """n pairs of parallel triangles, out of each other's reach."""
    from elastodynamicebem_b200 import mesh
    one = np.array([[0, 0, 0], [H, 0, 0], [0, H, 0], [0, 0, 0.5], [H, 0, 0.5], [0, H, 0.5]])
    x = np.concatenate([one + [4.0 * p, 0, 0] for p in range(n)])
    return mesh.Mesh(x, np.arange(6 * n).reshape(-1, 3))


def _params():
    from elastodynamicebem_b200 import problem
    prm = problem.ProblemParams(1, 1, 2, 1, 20)
    assert prm.velP == 2 and prm.velS == 1 and 5 * prm.dt == 0.25 and 10 * prm.dt == 0.5
    return prm


@pytest.mark.parametrize("n,rule", [(1, (12, 1, 12)), (128, (3, 1, 3))], ids=["warp", "thread"])
def test_ghc(oracle, n, rule):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import elastodynamicebem_b200.core as core
    m, prm = _pairs(n), _params()
    E = core.assemble_ghc(core.DeviceMesh(m), prm, *rule, 0, 20, sa_diagonal=False).cpu().numpy()
    Eo = oracle.assemble_ghc(m, prm, *rule, 0, 20)
    assert np.abs(E - Eo).max() <= TOL * np.abs(Eo).max()


@pytest.mark.parametrize("fix", [False, True])
def test_k(oracle, fix):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import elastodynamicebem_b200.core as core
    m, prm = _pairs(1), _params()
    dm = core.DeviceMesh(m)
    LK = core.num_blocks_dir(dm, prm)[1]
    K = core.assemble_k(dm, prm, 12, 1, 12, 0, 0, LK, fix=fix).cpu().numpy()
    Ko = oracle.assemble_k(m, prm, 12, 1, 12, 0, LK, nblocks=LK, fix=fix)
    assert np.abs(K - Ko).max() <= TOL * np.abs(Ko).max()


@pytest.mark.parametrize("speed", [1, 2])
@pytest.mark.parametrize("t,k", [(0.93, 12), (0.93, 14), (0.8, 12)])
def test_pp_dir(oracle, speed, t, k):
    """A receiver above a node at c (t - k dt), rounded as written."""
    if not cuda_available():
        pytest.skip("no CUDA device")
    import elastodynamicebem_b200.core as core
    m, prm = _pairs(1), _params()
    b = core.quad_gh(12)[0][4]
    x = np.array([H * b[1], H * b[2], speed * (t - k * prm.dt)])
    got = core.pp_dir_matrices(core.DeviceMesh(m), prm, 1, 12, x, t)
    want = oracle.pp_dir_matrices(m, prm, 1, 12, x, t)
    for a, b in zip(got, want):
        assert np.abs(a - b).max() <= TOL * np.abs(b).max()
