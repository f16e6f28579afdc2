"""The kNN's ways through the device against the oracle: one warp per query up
to 98,304 particles, one query per lane beyond, and what the latter hands over
or does twice (bins laid lower or finer, periodic images per pair, queries with
many particles at one distance).  Densities bit for bit; neighbour rows equal
except where distances tie exactly at the last place."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

SMALL = 98304  # largest set with one warp per query


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not gpu_available():
        pytest.skip("no CUDA device")
    from ahop_b200 import build
    build.build()


def _wrap(p, box):
    p = np.mod(p + 0.5 * box, box) - 0.5 * box
    p[p >= 0.5 * box] = -0.5 * box
    return p


def _clustered(n, rng, box):
    """Half uniform, half in clumps of very different sizes and densities."""
    k = n // 2
    c = (rng.random((40, 3)) - 0.5) * box
    r = 10.0 ** rng.uniform(-4.0, -1.0, 40) * box
    h = rng.integers(0, 40, k)
    p = np.concatenate([c[h] + r[h, None] * rng.normal(size=(k, 3)), (rng.random((n - k, 3)) - 0.5) * box])
    return _wrap(p[rng.permutation(n)], box)


def _corner(n, rng, box):
    """All but 60 particles in a clump over the box's corner (all eight periodic images)."""
    p = np.concatenate([1e-3 * box * rng.normal(size=(n - 60, 3)) + 0.5 * box, (rng.random((60, 3)) - 0.5) * box])
    return _wrap(p[rng.permutation(n)], box)


def _shells(n, rng, box):
    """Particles each with 150 others at one distance (to 1e-12), far from the rest."""
    m = 20
    c = (np.stack(np.meshgrid(np.arange(5), np.arange(2), np.arange(2), indexing="ij"), -1).reshape(-1, 3) - 2) * 0.05
    v = rng.normal(size=(m, 150, 3))
    v /= np.linalg.norm(v, axis=2, keepdims=True)
    s = np.concatenate([c, (c[:, None] + 2e-3 * v).reshape(-1, 3)])
    p = np.concatenate([s, rng.random((n - len(s), 3)) * 0.2 + 0.25])
    return _wrap(p[rng.permutation(n)] * box, box)


def _lattice(n, rng, box):
    """A jittered-free lattice: whole shells of (nearly) equal distances."""
    k = int(np.ceil(n ** (1.0 / 3.0)))
    p = (np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] / k - 0.5) * box
    return p[rng.permutation(n)]


@pytest.mark.parametrize("make,n,nv,box", [
    (_clustered, 33, 32, 1.0), (_clustered, 40, 32, 1.0), (_clustered, 1000, 2, 1.0), (_corner, 3001, 20, 100.0),
    (_shells, 5000, 32, 1.0), (_clustered, SMALL, 32, 1.0), (_clustered, SMALL + 1, 32, 1.0),
    (_clustered, 131103, 17, 100.0), (_corner, 100001, 32, 1.0), (_shells, 120007, 32, 1.0),
    (_lattice, 103823, 32, 1.0), (_lattice, 98400, 2, 7.0)])
def test_knn_matches_oracle(make, n, nv, box):
    import oracle
    from ahop_b200 import finder
    pos = make(n, np.random.default_rng(n + nv), box)
    mass = np.full(n, 1.0 / n)
    nhop = min(16, nv)
    finder.configure(n, box=box, nvoisins=nv, nhop=nhop)
    st = finder.run_stages(pos, mass, last_stage=2, store_neighbours=nv)
    if n <= 100:  # the oracle's cells need more particles: all pairs
        d = np.abs(pos[:, None] - pos[None])
        d = np.maximum(0.0, np.minimum(d, box - d))
        d2 = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
        np.fill_diagonal(d2, np.inf)
        nei = np.argsort(d2, axis=1, kind="stable")[:, :nv]
    else:
        ref = oracle.run(pos, mass, oracle.default_params(n, box=box, nvoisins=nv, nhop=nhop), capture_neighbours=nv)
        nei = ref["neighbours"]
        assert np.array_equal(st["density"], ref["density"])

    def dist2(rows):
        a = np.abs(pos[:, None, :] - pos[rows])
        a = np.maximum(0.0, np.minimum(a, box - a))
        return (a[..., 0] * a[..., 0] + a[..., 1] * a[..., 1]) + a[..., 2] * a[..., 2]

    mine = st["neighbours"] - 1
    dm = dist2(mine)
    assert np.array_equal(dm, np.sort(dist2(nei), axis=1))  # the same distances, ascending
    tie = dm[:, 1:] == dm[:, :-1]
    assert np.all(mine[:, 1:][tie] > mine[:, :-1][tie])     # equal ones by particle index
    assert np.all(mine != np.arange(n)[:, None])
    bad = np.nonzero((np.sort(mine, 1) != np.sort(nei, 1)).any(1))[0]
    for i in bad:  # only particles at exactly the last distance may differ
        only = np.setxor1d(mine[i], nei[i])
        a = np.abs(pos[only] - pos[i])
        a = np.maximum(0.0, np.minimum(a, box - a))
        assert np.all((a[:, 0] * a[:, 0] + a[:, 1] * a[:, 1]) + a[:, 2] * a[:, 2] == dm[i, -1])
