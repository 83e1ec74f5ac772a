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


def _traction_slices(oracle, m, prm, n_sub, n_sing, x, t):
    """P of kernelP.cu level by level in extended precision: the levels cancel in
    the second difference, which costs the 64-bit oracle 1e-11 of the largest entry
    next to the surface."""
    F = np.longdouble
    b, w = oracle.gauss_hammer(n_sing, n_sub)
    b, w = b.astype(F), np.tile(w.astype(F), n_sub)
    lam, mu, cP, cS, dt = (F(v) for v in (prm.lam, prm.mu, prm.velP, prm.velS, prm.dt))
    nhat = int(np.ceil(t / prm.dt))
    P = np.zeros((nhat + 2, 3, 3 * m.number_nodes), F)
    for tri in m.triangles:
        v = m.coordinates.astype(F)[tri]
        n = np.cross(v[1] - v[0], v[2] - v[0])
        area = np.sqrt((n * n).sum()) / 2
        n = n / (2 * area)
        X = x.astype(F) - b @ v
        r = np.sqrt((X * X).sum(1))
        ir, xn = (1 / r)[:, None, None], (X @ n)[:, None, None]
        A, XX, d = X[:, :, None] * n, X[:, :, None] * X[:, None, :], np.eye(3, dtype=F)
        B = np.swapaxes(A, 1, 2)
        for k in range(nhat + 1):
            tk = F(t) - k * dt
            if tk <= 0:
                continue
            tP, tS = 1 / ir / cP, 1 / ir / cS
            RP, RS = np.maximum(tk - tP, 0), np.maximum(tk - tS, 0)
            HP, HS = RP > 0, RS > 0
            SP, SS = RP * RP * (RP + 3 * tP) / 6, RS * RS * (RS + 3 * tS) / 6
            M = (lam * A * ir**2 + 2 * mu * xn * XX * ir**4) * HP / cP**3
            M = M + mu * (B * ir**2 + xn * (d * ir**2 - 2 * XX * ir**4)) * HS / cS**3
            M = M + ((lam - 2 * mu) * A - 2 * mu * B - 2 * mu * xn * (d - 6 * XX * ir**2)) * ir**3 * RP / cP**2
            M = M + mu * (2 * A + 3 * B + 3 * xn * (d - 4 * XX * ir**2)) * ir**3 * RS / cS**2
            M = M - 6 * mu * (A + B + xn * (d - 5 * XX * ir**2)) * ir**5 * (SP - SS)
            for c in range(3):
                P[k, :, 3 * tri[c]:3 * tri[c] + 3] += ((w * area * b[:, c])[:, None, None] * M).sum(0)
    D = (P[:-2] - 2 * P[1:-1] + P[2:]) / (4 * np.pi * prm.rho * dt)
    return D.reshape(3 * nhat, -1)


@pytest.mark.parametrize("rule,nT,t", [
    ((4, 3), 40, 0.013),         # before every arrival: zero exactly
    ((64, 7), 20, 0.6),          # chunks of 128 nodes
    ((4, 3), 160, 0.93),         # three windows of slices
    ((1, 3), 64, 1.0),           # time on the grid, 64 slices exactly
])
def test_pp_dir_front_bins(oracle, rule, nT, t):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import elastodynamicebem_b200.core as core
    from elastodynamicebem_b200 import mesh, problem
    m = mesh.icosphere(1)
    c = m.coordinates + np.random.default_rng(3).uniform(-0.02, 0.02, m.coordinates.shape) * m.lMin
    m = mesh.Mesh(c, m.triangles)
    prm = problem.ProblemParams(1, 1, 1, 1, nT)
    x = np.array([0.93, 0.21, 0.11])
    P = core.pp_dir_matrices(core.DeviceMesh(m), prm, *rule, x, t)[1]
    Po = _traction_slices(oracle, m, prm, *rule, x, t)
    # second differences of levels that grow like (t / dt)^3
    tol = TOL + 1e-15 * np.ceil(t * nT) ** 3
    assert P.shape == Po.shape
    assert np.abs(P - Po).max() <= tol * np.abs(Po).max()
