"""Inference of the quadrature selector (csrc/selector.cu) over window lengths
and pair counts around the edges of its groups (32 pairs), blocks (256 pairs),
batches (64 lags) and staged windows (96 lags): the class of every (pair, lag)
against the network in float64 (oracle) on the device's features.

Lags whose probability lies within 1e-3 of the threshold, or whose two largest
outputs do, may fall either way in FP32 and are left out."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu


def _classes(selector_oracle, core, dm, m, prm, params, threshold, lag0, nlag):
    import torch
    N = m.numberTriangles
    j, i, l = (a.ravel() for a in np.meshgrid(np.arange(N), np.arange(N), np.arange(lag0, lag0 + nlag), indexing="ij"))
    d = np.linalg.norm(m.center[j] - m.center[i], axis=1)
    h = m.maxL[j] + m.maxL[i]
    on = ((l - 1) * prm.velS * prm.dt < d + h) & ((l + 1) * prm.velP * prm.dt >= d - h)
    smp = torch.from_numpy(np.stack([i, j, l], 1).astype(np.int32)).cuda()
    x = core.selector_features(dm, prm, smp).cpu().numpy().astype(np.float64)
    swept = core.selector_sweeps(dm, prm, smp).cpu().numpy() != 0
    P = selector_oracle.unpack(params)
    a = np.maximum(x @ P["W1"].T + P["b1"], 0)
    z = np.maximum(a @ P["W2"].T + P["b2"], 0) @ P["W3"].T + P["b3"]
    pr = np.exp(z - z.max(1, keepdims=True))
    pr /= pr.sum(1, keepdims=True)
    top = np.sort(pr, 1)[:, ::-1]
    net = np.where(top[:, 0] >= threshold, pr.argmax(1), 3)
    sure = (np.abs(top[:, 0] - threshold) > 1e-3) & (top[:, 0] - top[:, 1] > 1e-3)
    return np.where(on, np.where(swept, 3, net), 0).reshape(N * N, nlag), (sure | swept | ~on).reshape(N * N, nlag), \
        (on & ~swept).sum()


@pytest.mark.parametrize("n,lag0,nlag,T", [(1, 0, 1, 0.5), (2, 0, 40, 2.0), (3, 0, 97, 5.0), (3, 5, 1, 2.0), (5, 0, 200, 8.0),
                                           (6, 3, 2, 1.0), (6, 0, 96, 6.0)])
def test_classes(n, lag0, nlag, T):
    if not cuda_available():
        pytest.skip("no CUDA device")
    import elastodynamicebem_b200.core as core
    import selector_oracle
    from elastodynamicebem_b200 import mesh, problem
    m = mesh.screen_graded(2 * n, 2 * n, 2.0) if n > 1 else mesh.screen_uniform(2)
    prm = problem.ProblemParams(1, 1, 2, T, 200)
    dm = core.DeviceMesh(m)
    params = core.selector_init(7)
    want, sure, asked = _classes(selector_oracle, core, dm, m, prm, params.cpu().numpy(), 0.3, lag0, nlag)
    cls, counts = core.selector_infer(params, dm, prm, 0.3, lag0, nlag)
    got = cls.cpu().numpy()
    assert np.all((got == want) | ~sure)
    assert sure.mean() > 0.9
    d = np.linalg.norm(m.center[:, None] - m.center[None], axis=2).ravel()
    assert sum(counts) == sum(int(((l - 1) * prm.velS * prm.dt < d + h).__and__((l + 1) * prm.velP * prm.dt >= d - h).sum())
                              for l in range(lag0, lag0 + nlag) for h in [(m.maxL[:, None] + m.maxL[None]).ravel()])
    assert counts[1] == int((got == 1).sum()) and counts[2] == int((got == 2).sum())
