"""One particle outside the box leaves the other leaves' search as it is: only
leaves that have a pair more than a box length apart are searched query by
query (the reference's distance is 0 along such an axis).  Rows and densities
of a sample, the queries near the opposite face among them, against all pairs."""
import numpy as np
import pytest

from conftest import gpu_available
from test_gpu_knn_scale import _counters

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not gpu_available():
        pytest.skip("no CUDA device")
    from ahop_b200 import build
    build.build()


@pytest.mark.parametrize("where,most", [((0.51, 0.1, -0.2), 0.1), ((-0.501, 0.7, 0.0), 0.5), ((0.3, 0.2, 0.1), 0.0)])
def test_outside_particle(where, most):
    from ahop_b200 import finder
    n = 131075
    rng = np.random.default_rng(11)
    pos = rng.random((n, 3)) - 0.5
    _, base = _counters(pos)
    pos[4321] = where
    _, c = _counters(pos)
    # uniform: leaves about 0.03 to 0.06 wide; those reaching the strip across
    # the box from the particle (0.01 wide; 0.001 and 0.2) come on top
    assert c["left"] <= base["left"] + most * c["leaves"] + 1, (c, base)
    assert c["queries_left"] <= base["queries_left"] + most * n + 32, (c, base)
    finder.configure(n)
    st = finder.run_stages(pos, np.full(n, 1.0 / n), last_stage=2, store_neighbours=32)
    far = np.argsort(np.abs(pos - np.asarray(where)).max(1))[-100:]  # across the box from it
    _check(pos, st, np.concatenate([[4321], far, rng.integers(0, n, 200)]))


def test_just_outside_the_faces():
    # a clump over the faces x = +-0.5 whose particles lie up to 4e-10 outside:
    # pairs across are more than a box length apart by 1 % of their distance
    from ahop_b200 import finder
    n, k = 120000, 4000
    rng = np.random.default_rng(12)
    pos = rng.random((n, 3)) - 0.5
    side = np.where(rng.random(k) < 0.5, 1.0, -1.0)
    pos[:k, 0] = side * (0.5 + 4e-10 * rng.random(k))
    pos[:k, 1:] = 0.2 + 1e-6 * rng.normal(size=(k, 2))
    pos = pos[rng.permutation(n)]
    finder.configure(n)
    st = finder.run_stages(pos, np.full(n, 1.0 / n), last_stage=2, store_neighbours=32)
    clump = np.nonzero(np.abs(pos[:, 0]) >= 0.5)[0]
    _check(pos, st, np.concatenate([rng.choice(clump, 200, replace=False), rng.integers(0, n, 50)]))


def _check(pos, st, queries):
    n = len(pos)
    rows = st["neighbours"] - 1
    for i in queries:
        d = np.abs(pos - pos[i])
        d = np.maximum(0.0, np.minimum(d, 1.0 - d))
        d2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
        d2[i] = np.inf
        want = np.lexsort((np.arange(n), d2))[:32]
        assert np.array_equal(rows[i], want), i
        r = 0.5 * np.sqrt(d2[want[-1]])
        u = np.sqrt(d2[want[:-1]]) / r
        w = np.where(u <= 1, 1 - 1.5 * u ** 2 + 0.75 * u ** 3, np.where(u <= 2, 0.25 * (2 - u) ** 3, 0.0))
        rho = (w.sum() + 1) / n / (float(np.float32(3.141592654)) * r ** 3)
        assert abs(st["density"][i] - rho) <= 1e-12 * rho
