"""The per-front closed form of the inner integral (csrc/sa_front.cuh) against
an edge quadrature (front_host/edge_quadrature.hpp) and the binary128 oracle, both compiled
for the host: every level, front and child state of meshes whose children are
thin, coplanar, collinear with a side, seen from inside, or scaled.

Tolerance, relative to the largest block: a block is a second difference of
F(t_k), which grows like t^2, so the rounding of F (some tens of units of
2.2e-16) enters times up to L^2: 50 * 2.2e-16 * 40^2 = 2e-11 for 40 levels,
4e-10 for 200.  Scales far from 1 are compared with the quadrature only: the
reference's 1e-6 thresholds make both differ from the exact value there."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from elastodynamicebem_b200 import core, mesh, problem

P = problem.ProblemParams


@pytest.fixture(scope="module")
def front(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("front") / "libfront.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fopenmp", "-fPIC", "-shared", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "elastodynamicebem_b200", "csrc"), "-o", so,
                    os.path.join(ROOT, "tests", "front_host", "front_host.cpp")], check=True)
    return C.CDLL(so)


def blocks(lib, m, prm, n_gh, src, fld, lag, closed):
    b, w = core.quad_gh(n_gh)
    out = np.zeros((len(src), 3, 3))
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)
    lib.front_blocks(ptr(m.coordinates), ptr(m.triangles), ptr(b), ptr(w), n_gh, C.c_double(prm.rho),
                     C.c_double(prm.velP), C.c_double(prm.velS), C.c_double(prm.dt), len(src), ptr(src), ptr(fld),
                     ptr(lag), int(closed), ptr(out))
    return out


def _jitter(m, h, seed=0, flat=False):
    rng = np.random.default_rng(seed)
    d = rng.uniform(-h, h, m.coordinates.shape)
    if flat:
        d[:, 2] = 0
    return mesh.Mesh(m.coordinates + d, m.triangles)


def _curved(n):
    m = mesh.screen_uniform(n)
    c = m.coordinates.copy()
    c[:, 2] = 0.2 * np.sin(3 * c[:, 0]) * c[:, 1]
    return mesh.Mesh(c, m.triangles)


CASES = [
    ("screen", mesh.screen_uniform(4), P(1, 1, 2, 1, 20), 7, True, 2e-11),
    ("screen_gh19", mesh.screen_uniform(3), P(1, 1, 2, 1, 20), 19, True, 2e-11),
    ("screen_jitter", _jitter(mesh.screen_uniform(4), 0.03, flat=True), P(1, 1, 2, 1, 40), 7, True, 2e-11),
    ("graded_sliver", mesh.screen_graded(8, 16, 3.0), P(1, 1, 2, 1, 40), 7, True, 2e-11),
    ("sphere", _jitter(mesh.icosphere(1), 0.05), P(1, 1, 1, 1, 40), 12, True, 2e-11),
    ("prism", mesh.prism_bar(1, 1, 3, 1.0), P(1, 1, 2, 2, 40), 7, True, 2e-11),
    ("curved", _curved(4), P(1, 1, 2, 1, 30), 3, True, 2e-11),
    ("equal_speeds", mesh.screen_uniform(4), P(1, 1, -1, 1, 8), 7, True, 2e-11),
    ("fine_dt", _jitter(mesh.icosphere(1), 0.05, 1), P(1, 1, 2, 1, 200), 7, True, 4e-10),
    ("one_step", mesh.screen_uniform(2), P(1, 1, 2, 1.5, 1), 7, True, 2e-11),
    ("small", _jitter(mesh.icosphere(1, 1e-2), 5e-4), P(1, 1, 2, 0.01, 40), 7, False, 2e-11),
    ("large", _jitter(mesh.screen_uniform(4, 500.0), 30.0), P(1, 1, 2, 1000, 20), 7, False, 2e-11),
]


@pytest.mark.parametrize("name,m,prm,n_gh,exact,tol", CASES, ids=[c[0] for c in CASES])
def test_closed_form(front, oracle, name, m, prm, n_gh, exact, tol):
    L = oracle.num_blocks(m, prm)
    rng = np.random.default_rng(5)
    q = 500
    src = rng.integers(0, m.numberTriangles, q).astype(np.int32)
    # a quarter of the pairs: the triangle itself; a quarter: one that shares a vertex
    fld = rng.integers(0, m.numberTriangles, q).astype(np.int32)
    fld[: q // 4] = src[: q // 4]
    inc = m.vertex_triangle_incidence().astype(int)
    near = inc.T @ inc > 0
    for k in range(q // 4, q // 2):
        fld[k] = rng.choice(np.flatnonzero(near[src[k]]))
    lag = rng.integers(0, L, q).astype(np.int32)
    lag[: q // 2: 2] = rng.integers(0, min(L, 6), len(lag[: q // 2: 2]))
    got = blocks(front, m, prm, n_gh, src, fld, lag, True)
    quad = blocks(front, m, prm, n_gh, src, fld, lag, False)
    scale = np.abs(quad).max()
    assert scale > 0 and np.isfinite(got).all()
    assert np.abs(got - quad).max() <= tol * scale
    if exact:
        ref = oracle.assemble_sa_pairs(m, prm, n_gh, src, fld, lag, variant="q")
        d, d0 = np.abs(got - ref).max(), np.abs(quad - ref).max()
        # where a front meets a node's distance exactly, the quadrature form shows what rounding decides there
        assert d <= max(tol * scale, 1.5 * d0)


def test_math(front):
    """Logarithm and first-quadrant arctangent: within 4 units of the last place of the long double functions (a
    series error of 1.3e-18 and some eight roundings, two of them of the full result)."""
    rng = np.random.default_rng(3)
    x = np.concatenate([10.0 ** rng.uniform(-12, 12, 20000), 1 + rng.uniform(-0.4, 0.6, 20000),
                        np.sqrt(0.5) * (1 + np.array([-2e-16, 0, 2e-16])), [1.0, 2.0, 0.5]])
    y = x * 10.0 ** rng.uniform(-10, 10, len(x))
    y[:1000] = x[:1000] * np.tan(np.pi / 8 * (1 + rng.uniform(-1e-15, 1e-15, 1000)))
    lg, at = np.empty_like(x), np.empty_like(x)
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)
    front.front_math(len(x), ptr(y), ptr(x), ptr(lg), ptr(at))
    rl, ra = np.log(x.astype(np.longdouble)), np.arctan2(y.astype(np.longdouble), x.astype(np.longdouble))
    eps = np.finfo(float).eps
    assert np.all(np.abs(lg - rl) <= 4 * eps * np.abs(rl))
    assert np.all(np.abs(at - ra) <= 4 * eps * ra)
    zero = np.zeros(1)
    front.front_math(1, ptr(np.ones(1)), ptr(zero), ptr(lg), ptr(at))
    assert abs(at[0] - np.pi / 2) <= eps
