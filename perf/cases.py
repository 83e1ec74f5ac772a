"""The calls whose time is measured, over the sizes a user of the library runs.

A user solves one problem on one surface mesh: assemble the space-time blocks
(semi-analytic, numerical-inner, or the direct formulation's V and K), march
in time, and evaluate the displacement at points.  Every case is one of those
calls on a mesh of the kinds the benchmark workloads use (flat and graded
screens, the icosphere, the prism bar), with the vertices moved by the seed so
that no front radius coincides with a mesh distance by symmetry.

``exact`` integrates the kernels by plain Gauss-Legendre quadrature in 64 bits
(or solves the marching recurrence with torch) where that is quick.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from elastodynamicebem_b200 import core, mesh as meshes, problem

DEV = "cuda"


# ---------------------------------------------------------------------------
# cases

def _c(name, kind, surface, a, b=0, **more):
    d = {"kind": kind, "surface": surface, "a": a, "b": b, "T": 1.0, "nT": 20, "lam": 2.0, "gh": 7}
    if name:
        d["name"] = name
    d.update(more)
    return d


def listed():
    return [
        # a convergence study's coarsest mesh: launches and host work count
        _c("sa_screen32_gh3", "sa", "screen", 4, 4, gh=3),
        # the prism bar with a higher outer rule, triangle count not a multiple of 32
        _c("sa_prism252_gh12", "sa", "prism", 3, nT=40),
        # an everyday mesh: one refinement below the headline sphere
        _c("sa_sphere320_gh7", "sa", "sphere", 2, nT=40, lam=1.0),
        # the headline benchmark: all 40 blocks of the 1280-triangle sphere
        _c("sa_sphere1280_gh7", "sa", "sphere", 3, nT=40, lam=1.0),
        # the whole indirect solve in one call (blocks, right-hand side, marching) on a screen
        _c("solve_screen286", "solve", "screen", 11, 13, nT=30),
        # block-sparse blocks and the marching on them, edge-graded screen, small time step
        _c("banded_graded480", "banded", "graded", 12, 20, nT=64),
        # marching on dense blocks at hand (many right-hand sides against one assembly)
        _c("march_prism700", "march", "prism", 5, nT=48),
        # numerical-inner assembly, the "GPU 7 16 3" method
        _c("ghc_sphere320_7_16_3", "ghc", "sphere", 2, nT=40, lam=1.0, n_sub=16, n_sing=3),
        # operators V and K of the direct formulation, "FN 7 4 3 16"
        _c("direct_vk_prism448", "vk", "prism", 4, T=0.8, nT=40, n_sub=4, n_sing=3, n_diag=16),
        # Neumann marching of the direct formulation and the displacement at interior points
        _c("dn_prism448", "dn", "prism", 4, T=0.8, nT=40, n_sub=4, n_sing=3, npts=16, ntimes=4),
        # closed-form post-processing: a cloud of points over the whole time grid
        _c("pp_sphere1280_256pts", "pp", "sphere", 3, nT=40, lam=1.0, npts=256, ntimes=40),
        # numerical post-processing: the time history of one receiver
        _c("ppnum_sphere320_1pt", "ppnum", "sphere", 2, nT=40, lam=1.0, n_sub=16, n_sing=3, npts=1, ntimes=40,
           layer=False),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _surface(rng, most):
    """A surface of at most `most` triangles (at least 18), sizes spread over their logarithm."""
    want = math.exp(rng.uniform(math.log(18), math.log(most)))
    kind = rng.choice(["screen", "graded", "sphere", "prism"])
    if kind == "screen":
        a = max(3, min(int(math.sqrt(most / 2)), int(round(math.sqrt(want / 2) * rng.uniform(0.7, 1.0)))))
        b = max(3, min(most // (2 * a), int(round(want / (2 * a)))))
        return kind, a, b
    if kind == "graded":
        a = 2 * max(2, min(int(math.sqrt(most / 8)), int(round(math.sqrt(want / 8) * rng.uniform(0.7, 1.0)))))
        b = 2 * max(2, min(most // (4 * a), int(round(want / (4 * a)))))
        return kind, a, b
    if kind == "sphere":
        k = max(k for k in range(0, 4) if 20 * 4 ** k <= max(20, min(most, 1.5 * want)))
        return kind, k, 0
    n = max(1, min(int(math.sqrt(most / 28)), int(round(math.sqrt(want / 28)))))
    return kind, n, 0


def draw(rng):
    kind = rng.choice(["sa", "sa", "sa", "solve", "banded", "march", "ghc", "vk", "dn", "pp", "ppnum"])
    most = {"sa": 1100, "solve": 700, "banded": 700, "march": 800, "ghc": 330, "vk": 450, "dn": 450, "pp": 1280,
            "ppnum": 700}[kind]
    surface, a, b = _surface(rng, most)
    if kind in ("vk", "dn"):
        surface, a, b = "prism", rng.choice([1, 2, 3, 4]), 0
    nT = _log_int(rng, 8, 44)
    more = {"nT": nT, "T": round(nT * rng.uniform(0.02, 0.035), 4), "lam": round(rng.uniform(0.5, 3.0), 3)}
    if kind in ("sa", "solve", "banded"):
        more["gh"] = rng.choice([3, 7, 7, 12]) if surface != "sphere" or a < 3 else rng.choice([3, 7])
    if kind in ("ghc", "vk", "dn", "ppnum"):
        more["n_sub"], more["n_sing"] = rng.choice([(4, 3), (4, 7), (16, 3)])
        if kind == "vk":
            more["n_sub"], more["n_sing"], more["n_diag"] = 4, 3, 16
    if kind == "pp":
        more.update(npts=_log_int(rng, 1, 256), ntimes=min(nT, _log_int(rng, 1, 40)))
    if kind == "ppnum":
        more["layer"] = rng.random() < 0.5
        more.update(npts=_log_int(rng, 1, 64), ntimes=1) if more["layer"] else more.update(
            npts=1, ntimes=min(nT, _log_int(rng, 2, 40)))
    if kind == "dn":
        more.update(npts=_log_int(rng, 1, 16), ntimes=rng.choice([1, 2, 4]))
    return _c(None, kind, surface, a, b, **more)


# ---------------------------------------------------------------------------
# inputs

def _mesh(case, seed):
    """The case's surface with vertices moved by the seed, up to 3 % of the local spacing."""
    rng = np.random.default_rng([11, seed])
    kind, a, b = case["surface"], case["a"], case["b"]
    if kind == "screen" or kind == "graded":
        ax = [np.linspace(-0.5, 0.5, n + 1) if kind == "screen" else meshes.graded_axis(n) for n in (a, b)]
        for x in ax:
            x[1:-1] += rng.uniform(-0.03, 0.03, len(x) - 2) * np.minimum(np.diff(x)[:-1], np.diff(x)[1:])
        return meshes.screen_from_axes(ax[0] * rng.uniform(0.97, 1.03), ax[1] * rng.uniform(0.97, 1.03), kind)
    if kind == "sphere":
        m = meshes.icosphere(a)
        x = m.coordinates + rng.uniform(-0.03, 0.03, m.coordinates.shape) * m.lMin
        return meshes.Mesh(x / np.linalg.norm(x, axis=1, keepdims=True), m.triangles, name="sphere")
    m = meshes.prism_bar(1.0, 1.0, 3.0, 1.0 / a)
    return meshes.Mesh(m.coordinates * rng.uniform(0.95, 1.05, 3), m.triangles, name="prism")


def _params(case):
    return problem.ProblemParams(1.0, 1.0, case["lam"], case["T"], case["nT"])


def _datum(case):
    return {"screen": problem.DATUM_SCREEN_T4EXP, "graded": problem.DATUM_SCREEN_T4EXP,
            "sphere": problem.DATUM_RADIAL_SIN, "prism": problem.DATUM_BAR_H3}[case["surface"]]


def _points(case, seed):
    """Receivers off the surface, near enough for the P front to arrive well within the run: above the screen,
    outside the sphere, inside the bar."""
    rng = np.random.default_rng([13, seed])
    n, p = case["npts"], _params(case)
    off = p.velP * p.Tfin * rng.uniform(0.1, 0.45, n)
    if case["surface"] == "sphere":
        d = rng.normal(size=(n, 3))
        return d / np.linalg.norm(d, axis=1, keepdims=True) * (1.0 + off[:, None])
    if case["surface"] == "prism":
        return np.column_stack([np.minimum(off, 0.8), rng.uniform(0.1, 0.9, n), rng.uniform(0.3, 2.7, n)])
    return np.column_stack([rng.uniform(-0.5, 0.5, (n, 2)), off])


def _times(case):
    """Output instants on the time grid, spread over it, the last one among them."""
    p = _params(case)
    return p.dt * np.unique(np.linspace(p.nT, 1, case["ntimes"]).round().astype(int))


def _field(rows, cols, seed):
    """A density as a marching leaves it: smooth growth in time, scatter over the unknowns (torch, rows x cols)."""
    rng = np.random.default_rng([17, seed])
    t = (np.arange(rows)[:, None] + 1.0) / rows
    v = np.sin(2 * math.pi * t * rng.uniform(0.5, 1.5, cols)) * rng.uniform(-1.0, 1.0, cols)
    return torch.from_numpy(np.ascontiguousarray(v)).to(DEV)


def _travel_blocks(rows_x, cols_x, size, params, L, diag, strength, seed):
    """Blocks shaped like a retarded operator's: E_l[3i + c, 3j + d] lives on the lags between the P and the S
    arrival, falls with the distance, and E_0's diagonal dominates.  (L, 3 rows, 3 cols), column-major storage."""
    g = torch.Generator(device=DEV).manual_seed(1000 + int(seed))
    r = torch.cdist(rows_x, cols_x)
    out = torch.empty((L, 3 * len(cols_x), 3 * len(rows_x)), dtype=torch.float64, device=DEV)
    noise = torch.rand((3 * len(cols_x), 3 * len(rows_x)), generator=g, dtype=torch.float64, device=DEV) - 0.5
    for l in range(L):
        lo, hi = r / params.velP, r / params.velS
        on = (((l + 1) * params.dt > lo - size) & ((l - 1) * params.dt < hi + size)).double() * strength / (r + size)
        out[l] = on.t().repeat_interleave(3, 0).repeat_interleave(3, 1) * noise / (1 + l)
    if diag is not None:
        out[0] += diag
    return out


def _march_inputs(case, seed):
    """(E storage, right-hand sides) of the dense marching."""
    p, m = _params(case), _mesh(case, seed)
    x = torch.from_numpy(m.center).to(DEV)
    E = _travel_blocks(x, x, float(m.maxL.mean()), p, _num_blocks(case, m), None, 1.0, seed)
    E[0] += 1.5 * E[0].abs().sum(1).max() * torch.eye(E.shape[1], dtype=torch.float64, device=DEV)
    return E, _field(p.nT, 3 * m.numberTriangles, seed)


def _dn_inputs(case, seed):
    """(V, K, gV) of the Neumann marching: V as an assembly leaves it, K_0 a quarter of the identity term."""
    p, m = _params(case), _mesh(case, seed)
    xc, xv = torch.from_numpy(m.center).to(DEV), torch.from_numpy(m.coordinates).to(DEV)
    L = _num_blocks(case, m)
    size = float(m.maxL.mean())
    G = _identity_term(m)
    scale = float(m.area.mean())
    V = _travel_blocks(xc, xc, size, p, L, None, scale * 0.02, seed)
    K = _travel_blocks(xc, xv, size, p, L, 0.25 * G.t(), scale * 0.002, seed + 7)
    return V.transpose(1, 2), K.transpose(1, 2), _field(p.nT, 3 * m.numberTriangles, seed), G


def _identity_term(m):
    """kron((vertex in triangle) area / 6, eye(3)), 3N x 3Nv."""
    inc = torch.from_numpy(m.vertex_triangle_incidence().T.astype(np.float64)).to(DEV)
    inc = inc * torch.from_numpy(m.area / 6).to(DEV)[:, None]
    return torch.kron(inc.contiguous(), torch.eye(3, dtype=torch.float64, device=DEV))


def _num_blocks(case, m):
    p = _params(case)
    x = torch.from_numpy(m.coordinates)
    return min(p.nT, math.ceil(float(torch.cdist(x, x).max()) / (p.velS * p.dt)) + 1)


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, s.prm = case, _params(case)
    kind = case["kind"]
    m = _mesh(case, seed)
    if kind == "march":
        E, s.b = _march_inputs(case, seed)
        s.E = E.transpose(1, 2)
        return s
    s.dm = core.DeviceMesh(m)
    if kind in ("sa", "ghc"):
        s.L = core.num_blocks(s.dm, s.prm)
    elif kind in ("solve", "banded"):
        s.datum = _datum(case)
    elif kind == "dn":
        s.V, s.K, s.g, _ = _dn_inputs(case, seed)
        s.pts, s.times = _points(case, seed), _times(case)
    elif kind in ("pp", "ppnum"):
        s.phi = _field(s.prm.nT, 3 * m.numberTriangles, seed)
        s.pts, s.times = _points(case, seed), _times(case)
    return s


# ---------------------------------------------------------------------------
# one pass

def run(s):
    c, kind = s.case, s.case["kind"]
    if kind == "sa":
        return core.assemble_sa(s.dm, s.prm, c["gh"], 0, s.L)
    if kind == "solve":
        return core.timemarch_sa(s.dm, s.prm, c["gh"], s.datum)[0]
    if kind == "banded":
        op = core.BandedOperator(s.dm, s.prm, c["gh"])
        phi = op.march(core.rhs(s.dm, s.prm, c["gh"], s.datum))
        op.close()
        return phi
    if kind == "march":
        return core.march(s.E, s.b)
    if kind == "ghc":
        return core.assemble_ghc(s.dm, s.prm, c["gh"], c["n_sub"], c["n_sing"], 0, s.L)
    if kind == "vk":
        return (core.assemble_v(s.dm, s.prm, c["gh"], c["n_sub"], c["n_sing"], c["n_diag"]),
                core.assemble_k(s.dm, s.prm, c["gh"], c["n_sub"], c["n_sing"], c["n_diag"]))
    if kind == "dn":
        u = core.march_dn(s.dm, s.prm, s.V, s.K, s.g)
        return u, core.pp_dir(s.dm, s.prm, c["n_sub"], c["n_sing"], s.g, u, s.pts, s.times, fix=True)
    if kind == "pp":
        return core.pp_sa(s.dm, s.prm, s.phi, s.pts, s.times)
    if kind == "ppnum":
        return core.pp_gpu(s.dm, s.prm, s.phi, s.pts, s.times, c["n_sub"], c["n_sing"],
                           core.PP_LAYER if c["layer"] else core.PP_POINT)
    raise ValueError(kind)


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _pair_lags(case, m):
    """Non-null (source, field, lag) blocks of the null test."""
    p, L = _params(case), _num_blocks(case, m)
    d = np.sqrt(((m.center[:, None] - m.center[None]) ** 2).sum(-1))
    h = m.maxL[:, None] + m.maxL[None]
    lo = np.ceil((d - h) / (p.velP * p.dt) - 1)
    hi = np.ceil((d + h) / (p.velS * p.dt) + 1) - 1
    return float(np.clip(np.minimum(hi, L - 1) - np.maximum(lo, 0) + 1, 0, None).sum())


def work(case):
    p, m, kind = _params(case), _mesh(case, 0), case["kind"]
    N, Nv, L, gh = m.numberTriangles, m.number_nodes, _num_blocks(case, m), case["gh"]
    n3 = 3.0 * N
    mesh_bytes = 24.0 * Nv + 12.0 * N
    # a closed-form inner integral of one (outer node, field triangle, instant): 3 sides, about 100 operations each
    closed = 300.0
    # an evaluation of the integrated kernel at one pair of nodes: about 40 operations
    node = 40.0
    march = 2.0 * n3 ** 3 / 3 + 2.0 * n3 * n3 * sum(min(n, L - 1) + 1 for n in range(p.nT))
    if kind == "sa":
        return {"bytes": mesh_bytes + 8 * n3 * n3 * L, "flops": _pair_lags(case, m) * gh * closed}
    if kind == "solve":
        return {"bytes": mesh_bytes + 8 * n3 * p.nT, "flops": _pair_lags(case, m) * gh * closed + march}
    if kind == "banded":
        pl = _pair_lags(case, m)
        return {"bytes": mesh_bytes + 8 * n3 * p.nT, "flops": pl * gh * closed + 2 * n3 ** 3 / 3 + 18.0 * pl * p.nT / 2}
    if kind == "march":
        return {"bytes": 8 * (n3 * n3 * L + 2 * n3 * p.nT), "flops": march}
    inner = case.get("n_sub", 1) * case.get("n_sing", 1)
    if kind == "ghc":
        return {"bytes": mesh_bytes + 8 * n3 * n3 * L, "flops": float(N) * N * gh * inner * 2 * node}
    if kind == "vk":
        pairs = float(N) * N * gh * inner
        return {"bytes": mesh_bytes + 8 * n3 * L * (n3 + 3 * Nv), "flops": pairs * node * (2 + 3 * 2 * 2)}
    if kind == "dn":
        nv3 = 3.0 * Nv
        steps = 2.0 * n3 * (n3 + nv3) * sum(min(n + 1, L) for n in range(p.nT))
        field = case["npts"] * float(sum(round(t / p.dt) for t in _times(case))) * N * inner * node * 4
        return {"bytes": 8 * (n3 * L * (n3 + nv3) + (n3 + nv3) * p.nT), "flops": 4 * n3 * nv3 * nv3 + steps + field}
    npts, times = case["npts"], _times(case)
    one = closed if kind == "pp" else inner * node
    inst = len(set(int(round(t / p.dt)) - k for t in times for k in range(p.nT) if round(t / p.dt) > k))
    pairs = sum(round(t / p.dt) for t in times)
    return {"bytes": mesh_bytes + 8 * (n3 * p.nT + 3.0 * npts * (len(times) + 1)),
            "flops": float(N) * npts * (inst * one / 4 + 18.0 * pairs / 4)}


# ---------------------------------------------------------------------------
# 64-bit values by plain quadrature

def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return torch.from_numpy(x).to(DEV), torch.from_numpy(w).to(DEV)


def _rule(n, n_sub=1):
    """The 3- or 7-point Gauss-Hammer rule of degree 2 or 5 on n_sub congruent sub-triangles: barycentric nodes,
    weights summing to 1; None for others."""
    if n == 3:
        b, w = [[2 / 3, 1 / 6, 1 / 6]], [1 / 3]
    elif n == 7:
        q = math.sqrt(15.0)
        lo, hi = (6 - q) / 21, (6 + q) / 21
        b, w = [[1 - 2 * lo, lo, lo], [1 - 2 * hi, hi, hi]], [(155 - q) / 1200, (155 + q) / 1200]
    else:
        return None
    nodes, weights = ([[1 / 3] * 3], [9 / 40]) if n == 7 else ([], [])
    for t, v in zip(b, w):
        nodes += [t, [t[1], t[0], t[1]], [t[1], t[1], t[0]]]
        weights += [v] * 3
    k = int(round(math.sqrt(n_sub)))
    all_nodes = []
    for i in range(k):
        for j in range(k - i):
            up = np.array([[i, j], [i + 1, j], [i, j + 1]]) / k
            tris = [up] if i + j + 1 >= k else [up, np.array([[i + 1, j + 1], [i, j + 1], [i + 1, j]]) / k]
            for tri in tris:
                full = np.column_stack([tri, 1 - tri.sum(1)])
                all_nodes.append(np.array(nodes) @ full)
    return (torch.from_numpy(np.concatenate(all_nodes)).to(DEV),
            torch.from_numpy(np.tile(weights, n_sub) / n_sub).to(DEV))


def _inner(x, P, p, t):
    """S I + T of the closed-form inner integrals, halved: points x (Q, 3), triangles P (Q, 3, 3), instants t (K,)
    -> (K, Q, 3, 3), by Gauss-Legendre along each side as seen from the projected point."""
    e1 = P[:, 1] - P[:, 0]
    e1 = e1 / e1.norm(dim=1, keepdim=True)
    n = torch.linalg.cross(P[:, 0] - P[:, 2], P[:, 1] - P[:, 2])
    n = n / n.norm(dim=1, keepdim=True)
    e2 = torch.linalg.cross(n, e1)
    h = ((x - P[:, 0]) * n).sum(1)                                     # signed height of the point
    h = torch.where(h.abs() < 1e-6, torch.zeros_like(h), h)
    z = h.abs()
    d = P - (x - ((x - P[:, 0]) * n).sum(1, keepdim=True) * n)[:, None]
    tri = torch.stack([(d * e1[:, None]).sum(2), (d * e2[:, None]).sum(2)], 2)
    gx, gw = _gauss(12)
    at = (torch.arange(8, device=x.device)[:, None] + 0.5 + 0.5 * gx).reshape(-1)     # eight sub-pieces of a piece
    gw = gw.repeat(8)
    cP, cS = p.velP, p.velS
    k1, k5, k6 = 1 / cP ** 2, 1 / cP ** 2 + 1 / cS ** 2, 1 / cS ** 2 - 1 / cP ** 2
    out = torch.zeros((len(t), len(x), 3, 3), dtype=torch.float64, device=x.device)
    for ti, tt in enumerate(t.tolist()):
        rP, rS = cP * tt, cS * tt
        M = torch.zeros((len(x), 3, 3), dtype=torch.float64, device=x.device)
        S = torch.zeros(len(x), dtype=torch.float64, device=x.device)
        fP = torch.sqrt(torch.clamp(rP * rP - z * z, min=0))          # in-plane front radii
        fS = torch.sqrt(torch.clamp(rS * rS - z * z, min=0))
        for c in range(3):
            A, B = tri[:, c], tri[:, (c + 1) % 3]
            u = B - A
            u = u / u.norm(dim=1, keepdim=True)
            F = A[:, 0] * u[:, 1] - A[:, 1] * u[:, 0]                    # signed distance of the side's line
            sgn, F = torch.sign(F), F.abs().clamp(min=1e-9)
            foot = torch.stack([u[:, 1], -u[:, 0]], 1) * sgn[:, None]    # unit vector to the foot
            sa, sb = torch.asinh((A * u).sum(1) / F), torch.asinh((B * u).sum(1) / F)
            cuts = [sa, sb]
            for f in (fP, fS):
                q = torch.acosh(torch.clamp(f / F, min=1.0))
                cuts += [torch.minimum(torch.maximum(q, sa), sb), torch.minimum(torch.maximum(-q, sa), sb)]
            cuts = torch.sort(torch.stack(cuts), 0).values
            for k in range(5):
                lo, step = cuts[k], (cuts[k + 1] - cuts[k]) / 8
                s = lo[:, None] + step[:, None] * at
                ch = torch.cosh(s)
                w = gw * 0.5 * step[:, None] / ch * sgn[:, None]     # d theta, oriented
                R = F[:, None] * ch
                cx = (foot[:, None, 0] + torch.sinh(s) * u[:, None, 0]) / ch
                cy = (foot[:, None, 1] + torch.sinh(s) * u[:, None, 1]) / ch
                zz = z[:, None]
                up, mid = torch.minimum(R, fP[:, None]), torch.minimum(R, fS[:, None])
                zero = torch.zeros_like(up)

                def radial(rho):
                    r = torch.sqrt(rho * rho + zz * zz).clamp(min=1e-300)
                    ir = 1 / r
                    flat = zz <= 0
                    C2 = torch.where(flat, zero, torch.log((rho + r).clamp(min=1e-300)) - rho * ir)
                    C4 = torch.where(flat, zero, -(r * r + r * rho + rho * rho) * ir ** 3 / (3 * (r + rho)))
                    z2 = zz * zz
                    return (r, -ir, r + z2 * ir, C2, -z2 * ir, -ir + z2 * ir ** 3 / 3, C4, -z2 * ir ** 3 / 3)
                a, b, o = radial(up), radial(mid), radial(zero)
                t2, on = tt * tt, (up > mid).double()
                sc = on * (k1 * (a[0] - b[0]) - t2 * (a[1] - b[1]))
                pl = on * (-k1 * (a[2] - b[2]) + 3 * t2 * (a[5] - b[5]))
                mx = on * (-k1 * (a[3] - b[3]) + 3 * t2 * (a[6] - b[6]))
                nn = on * (-k1 * (a[4] - b[4]) + 3 * t2 * (a[7] - b[7]))
                on = (mid > 0).double()
                sc = sc + on * k5 * (b[0] - torch.where(zz <= 0, zero, o[0]))
                pl = pl + on * k6 * (b[2] - torch.where(zz <= 0, zero, o[2]))
                mx = mx + on * k6 * (b[3] - o[3])
                nn = nn + on * k6 * (b[4] - torch.where(zz <= 0, zero, o[4]))
                S += (w * sc).sum(1)
                M[:, 0, 0] += (w * pl * cx * cx).sum(1)
                M[:, 0, 1] += (w * pl * cx * cy).sum(1)
                M[:, 1, 1] += (w * pl * cy * cy).sum(1)
                M[:, 0, 2] += (w * -h[:, None] * mx * cx).sum(1)
                M[:, 1, 2] += (w * -h[:, None] * mx * cy).sum(1)
                M[:, 2, 2] += (w * nn).sum(1)
        M[:, 1, 0], M[:, 2, 0], M[:, 2, 1] = M[:, 0, 1], M[:, 0, 2], M[:, 1, 2]
        C = torch.stack([e1, e2, n], 1)
        out[ti] = 0.5 * (C.transpose(1, 2) @ M @ C + S[:, None, None] * torch.eye(3, dtype=torch.float64, device=x.device))
    return out


def _exact_sa(case, seed):
    p, m = _params(case), _mesh(case, seed)
    N, L, gh = m.numberTriangles, _num_blocks(case, m), case["gh"]
    if float(N) * N * gh * L > 4e6 or _rule(gh) is None:
        return None
    P = torch.from_numpy(m.coordinates[m.triangles]).to(DEV)
    b, w = _rule(gh)
    nodes = torch.einsum("gv,nvc->ngc", b, P)                            # outer nodes (N, gh, 3)
    t = p.dt * torch.arange(1, L + 1, dtype=torch.float64)
    area = torch.from_numpy(m.area).to(DEV)
    x = nodes[:, None].expand(N, N, gh, 3).reshape(-1, 3)
    T = P[None, :, None].expand(N, N, gh, 3, 3).reshape(-1, 3, 3)
    F = torch.zeros((L + 2, N, N, 3, 3), dtype=torch.float64, device=DEV)   # levels -1, 0, 1, ..: shifted by one
    F[2:] = torch.einsum("i,g,lijgrc->lijrc", area, w, _inner(x, T, p, t).view(L, N, N, gh, 3, 3))
    E = (F[2:] - 2 * F[1:-1] + F[:-2]) / (4 * math.pi * p.rho)
    return E.permute(0, 1, 3, 2, 4).reshape(L, 3 * N, 3 * N)


def _exact_pp(case, seed):
    p, m = _params(case), _mesh(case, seed)
    times, pts = _times(case), torch.from_numpy(_points(case, seed)).to(DEV)
    N, Q, nT = m.numberTriangles, case["npts"], case["nT"]
    if float(N) * Q * nT > 4e6:
        return None
    P = torch.from_numpy(m.coordinates[m.triangles]).to(DEV)
    x, T = pts[:, None].expand(Q, N, 3).reshape(-1, 3), P[None].expand(Q, N, 3, 3).reshape(-1, 3, 3)
    M = torch.zeros((nT + 1, Q, 3, 3 * N), dtype=torch.float64, device=DEV)
    M[1:] = _inner(x, T, p, p.dt * torch.arange(1, nT + 1, dtype=torch.float64)).view(nT, Q, N, 3, 3).permute(
        0, 1, 3, 2, 4).reshape(nT, Q, 3, 3 * N) / (4 * math.pi * p.rho)
    phi = _field(nT, 3 * N, seed)
    u = torch.zeros((len(times), Q, 3), dtype=torch.float64, device=DEV)
    for q, t in enumerate(times):
        n = int(round(t / p.dt))
        for k in range(n):                                              # density of step k acts on [k dt, (k+1) dt]
            u[q] += (M[n - k] - M[n - k - 1]) @ phi[k]
    return u


def _exact_march(case, seed):
    E, b = _march_inputs(case, seed)
    E = E.transpose(1, 2)
    lu, piv = torch.linalg.lu_factor(E[0].contiguous())
    phi = torch.zeros_like(b)
    for n in range(len(b)):
        r = b[n].clone()
        for l in range(1, min(n, len(E) - 1) + 1):
            r -= E[l] @ phi[n - l]
        phi[n] = torch.linalg.lu_solve(lu, piv, r[:, None])[:, 0]
    return phi


def _exact_dn(case, seed):
    V, K, g, G = _dn_inputs(case, seed)
    A = K[0] + G
    q, r = torch.linalg.qr(A)
    u = torch.zeros((len(g), A.shape[1]), dtype=torch.float64, device=DEV)
    for n in range(len(g)):
        b = G @ u[n - 1] if n else torch.zeros(A.shape[0], dtype=torch.float64, device=DEV)
        for l in range(min(n + 1, len(V))):
            b = b + V[l] @ g[n - l]
        for l in range(1, min(n, len(K) - 1) + 1):
            b = b - K[l] @ u[n - l]
        u[n] = torch.linalg.solve_triangular(r, (q.T @ b)[:, None], upper=True)[:, 0]
    return u, None


def _exact_ghc(case, seed):
    """Off-diagonal blocks by the numerical rule, instant by instant; diagonal blocks by _inner."""
    p, m = _params(case), _mesh(case, seed)
    N, L, gh = m.numberTriangles, _num_blocks(case, m), case["gh"]
    if float(N) * N * gh * case["n_sub"] * case["n_sing"] * L > 6e9:
        return None
    P = torch.from_numpy(m.coordinates[m.triangles]).to(DEV)
    area = torch.from_numpy(m.area).to(DEV)
    b, w = _rule(gh)
    bi, wi = _rule(case["n_sing"], case["n_sub"])
    X, Y = torch.einsum("gv,nvc->ngc", b, P), torch.einsum("gv,nvc->ngc", bi, P)
    E = torch.zeros((L, N, 3, N, 3), dtype=torch.float64, device=DEV)
    eye = torch.eye(3, dtype=torch.float64, device=DEV)
    cP2, cS2 = p.velP ** 2, p.velS ** 2
    for o in range(gh):
        for q in range(len(bi)):
            x = Y[None, :, q] - X[:, None, o]
            r2 = (x * x).sum(2)
            r2[torch.arange(N), torch.arange(N)] = 1.0
            r = torch.sqrt(r2)
            wt = (w[o] * area)[:, None] * (wi[q] * area)[None]
            wt[torch.arange(N), torch.arange(N)] = 0.0
            K = []
            for k in range(-1, L + 1):
                t = k * p.dt
                if k < 1:
                    K.append(None)
                    continue
                HP, HS = (t - r / p.velP > 0).double(), (t - r / p.velS > 0).double()
                tail = (t * t - r2 / cP2) * HP - (t * t - r2 / cS2) * HS
                K.append((wt * ((HP / cP2 - HS / cS2) / r ** 3 + 1.5 * tail / r ** 5),
                          wt * (HS / cS2 / r - 0.5 * tail / r ** 3)))
            for l in range(L):
                g1 = g2 = 0.0
                for j, c in ((l + 2, 1.0), (l + 1, -2.0), (l, 1.0)):
                    if K[j] is not None:
                        g1, g2 = g1 + c * K[j][0], g2 + c * K[j][1]
                if torch.is_tensor(g1):
                    E[l] += (g1[:, :, None, None] * x[:, :, :, None] * x[:, :, None] +
                             g2[:, :, None, None] * eye).permute(0, 2, 1, 3)
    E /= 4 * math.pi * p.rho
    # the diagonal blocks, closed form
    t = p.dt * torch.arange(1, L + 1, dtype=torch.float64)
    F = torch.zeros((L + 2, N, 3, 3), dtype=torch.float64, device=DEV)
    for g in range(gh):
        F[2:] += (w[g] * area)[None, :, None, None] * _inner(X[:, g].contiguous(), P, p, t)
    D = (F[2:] - 2 * F[1:-1] + F[:-2]) / (4 * math.pi * p.rho)
    i = torch.arange(N, device=DEV)
    E[:, i, :, i, :] = D.permute(1, 0, 2, 3)
    return E.reshape(L, 3 * N, 3 * N)


def exact(case, seed):
    make = {"sa": _exact_sa, "pp": _exact_pp, "march": _exact_march, "dn": _exact_dn, "ghc": _exact_ghc}.get(case["kind"])
    return make(case, seed) if make else None
