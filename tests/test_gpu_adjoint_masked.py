"""The density adjoint with particles that have no upstream gradient: whatever
their positions (NaN, infinite) and lists hold, they add nothing, the other
gradients are the same bits as without them, and nothing is written past the
last row."""
import ctypes as C

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


@pytest.mark.parametrize("n,nv", [(31, 4), (33, 32), (97, 5), (1001, 33), (32769, 6)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_masked(n, nv, bad):
    import torch
    from ahop_b200 import _lib, autograd
    lib = autograd._bind()
    rng = np.random.default_rng(n + nv)
    # active particles only list active ones; no two contribute to one target
    # in the same order twice, so sums are compared with a margin below
    masked = rng.random(n) < 0.3
    masked[[0, n - 1]] = True
    live = np.nonzero(~masked)[0]
    pos = rng.random((n, 3)) - 0.5
    nei = np.zeros((n, nv), np.int32)
    for i in range(n):
        c = rng.choice(live, nv + 1, replace=len(live) <= nv)
        c = c[c != i][:nv]
        c = np.resize(c, nv)
        d = pos[c] - pos[i]
        d -= np.round(d)
        nei[i] = c[np.argsort((d * d).sum(1), kind="stable")]
    g = np.where(masked, 0.0, rng.normal(size=n))
    mass = np.ones(n)
    guard = 64
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    prm = autograd.AhopAdjParams(nv, 0, 1.0, 1.0, 1.0)

    def run(p, m, lists):
        out = torch.zeros((n + guard, 3), dtype=torch.float64, device="cuda")
        a = (t(p), t(m), t(lists), t(g))
        _lib.check(lib.ahop_density_adjoint(C.byref(prm), a[0].data_ptr(), a[1].data_ptr(), a[2].data_ptr(), n,
                                            a[3].data_ptr(), out.data_ptr(), None), "density_adjoint")
        torch.cuda.synchronize()
        return out.cpu().numpy()

    want = run(pos, mass, nei)
    pos2, mass2, nei2 = pos.copy(), mass.copy(), nei.copy()
    pos2[masked] = bad
    mass2[masked] = bad
    nei2[masked] = rng.integers(0, n, (int(masked.sum()), nv))  # masked rows may list masked particles
    got = run(pos2, mass2, nei2)
    assert np.all(got[n:] == 0.0)
    assert np.all(got[:n][masked] == 0.0) and np.all(want[:n][masked] == 0.0)
    # the same terms, in another order from run to run: one rounding per term
    count = np.bincount(nei[live].ravel(), minlength=n) + 2 * nv + 2
    scale = np.abs(want[:n]).max() if n > 1 else 1.0
    assert np.all(np.isfinite(got))
    assert np.all(np.abs(got[:n] - want[:n]) <= count[:, None] * 2.0 ** -52 * scale * nv)
