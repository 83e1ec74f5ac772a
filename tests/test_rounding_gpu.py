"""Rounding of the semi-analytic blocks on the device: no larger than that of
an integration of the same quantity that has no cancellation between the
fronts, the edge quadrature of tests/front_host, both against binary128.

Compared in the mean square over blocks of near and far pairs at all lags.
Both add terms of the same sizes (a front's radius times an angle, side
integrals), so their rounding is alike but for the functions: the device's err by
up to two units of the last place, the host's by one half to one.  Hence a factor
of 3.  (With the constants t^2 / F of both fronts added and subtracted the
device's blocks were off by 4 to 5 times the quadrature's on thin children.)"""
import numpy as np
import pytest

from conftest import cuda_available
from test_front_cpu import CASES, blocks, front  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,m,prm,n_gh,tol", [c[:4] + c[5:] for c in CASES if c[4]],
                         ids=[c[0] for c in CASES if c[4]])
def test_blocks(front, oracle, name, m, prm, n_gh, tol):  # noqa: F811
    if not cuda_available():
        pytest.skip("no CUDA device")
    import elastodynamicebem_b200.core as core
    dm = core.DeviceMesh(m)
    L = core.num_blocks(dm, prm)
    rng = np.random.default_rng(5)
    q = 1500
    src, fld = (rng.integers(0, m.numberTriangles, q).astype(np.int32) for _ in range(2))
    fld[: q // 4] = src[: q // 4]
    lag = rng.integers(0, L, q).astype(np.int32)
    E = core.assemble_sa(dm, prm, n_gh, 0, L).cpu().numpy().reshape(L, m.numberTriangles, 3, m.numberTriangles, 3)
    ref = oracle.assemble_sa_pairs(m, prm, n_gh, src, fld, lag, variant="q")
    rms = lambda d: np.sqrt((d ** 2).mean())
    dev, quad = rms(E[lag, src, :, fld] - ref), rms(blocks(front, m, prm, n_gh, src, fld, lag, False) - ref)
    # 2^-53 of the largest block: where the quadrature's own rounding is below it
    assert dev <= 3 * max(quad, 1.1e-16 * np.abs(ref).max())
