"""The fixed-list density and its adjoint against 64-bit torch where the kernels
change course: warps and blocks that are not full, lists shorter and longer
than a warp, particle rows packed from 32,768 particles on, gradients that are
zero for some particles, coincident neighbours."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not gpu_available():
        pytest.skip("no CUDA device")
    from ahop_b200 import build
    build.build()


@pytest.mark.parametrize("n,nv", [(2, 2), (33, 2), (129, 5), (1000, 32), (32767, 8), (32768, 33), (32801, 40)])
def test_density_and_adjoint(n, nv):
    import torch
    from ahop_b200 import autograd
    rng = np.random.default_rng(n * 100 + nv)
    pos = rng.random((n, 3)) - 0.5
    mass = rng.uniform(0.5, 1.5, n)
    if n > 1000:
        pos[7] = pos[6]  # coincident with a neighbour of its own
    nei = (np.arange(n)[:, None] + 1 + rng.permuted(np.tile(np.arange(max(n - 1, nv)), (min(n, 8), 1)),
                                                    axis=1)[np.arange(n) % min(n, 8), :nv]) % n
    if n > 1000:
        nei[6, 0] = 7
    d = pos[nei] - pos[:, None]
    d -= np.round(d)
    order = np.argsort((d * d).sum(2), axis=1, kind="stable")
    nei = np.take_along_axis(nei, order, 1).astype(np.int32)
    d = np.take_along_axis(d, order[..., None], 1)
    g = np.where(rng.random(n) < 0.2, 0.0, rng.normal(size=n))
    dev = torch.device("cuda:0")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    p = t(pos).requires_grad_(True)
    rho = autograd.SPHDensity.apply(p, t(mass), t(nei), 1.0)
    rho.backward(t(g))
    # the same sums in NumPy
    r = np.sqrt((d * d).sum(2))
    h = 0.5 * r[:, -1]
    u = r[:, :-1] / h[:, None]
    w = np.where(u <= 1, 1 - 1.5 * u ** 2 + 0.75 * u ** 3, np.where(u <= 2, 0.25 * (2 - u) ** 3, 0.0))
    dw = np.where(u <= 1, -3 * u + 2.25 * u ** 2, np.where(u <= 2, -0.75 * (2 - u) ** 2, 0.0))
    m = mass[nei[:, :-1]]
    C = 1.0 / float(np.float32(3.141592654))
    s = (m * w).sum(1) + mass
    want = C * s / h ** 3
    assert np.all(np.abs(rho.detach().cpu().numpy() - want) <= 1e-14 * nv * want)
    coef = np.empty((n, nv))
    coef[:, :-1] = g[:, None] * C * m * dw / h[:, None] ** 4
    coef[:, -1] = g * 0.5 * C * (-(m * dw * r[:, :-1]).sum(1) / h ** 5 - 3 * s / h ** 4)
    with np.errstate(divide="ignore", invalid="ignore"):
        v = np.where(r[..., None] > 0, coef[..., None] * d / r[..., None], 0.0)
    grad, size = np.zeros((n, 3)), np.zeros((n, 3))
    np.add.at(grad, nei, v)
    np.add.at(size, nei, np.abs(v))
    grad -= v.sum(1)
    size += np.abs(v).sum(1)
    # a few roundings per term, and the last term's own sum of nv terms
    assert np.all(np.abs(p.grad.cpu().numpy() - grad) <= 1e-14 * (nv + 20) * (size + np.abs(v[:, -1])) + 1e-14 * nv *
                  size.max())
