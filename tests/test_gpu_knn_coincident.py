"""Neighbour rows of particles with more coincident partners than neighbours:
at distance 0 too the row holds the smallest particle indices, whichever way
through the device a query takes (one warp per query up to 98,304 particles,
one query per lane beyond, and what that hands over)."""
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


@pytest.mark.parametrize("n,nv", [(20000, 32), (98304, 7), (98400, 32), (120011, 17)])
def test_coincident_rows(n, nv):
    from ahop_b200 import finder
    rng = np.random.default_rng(n + nv)
    pos = rng.random((n, 3)) - 0.5
    clump = np.full(n, -1)
    q = 0
    for c, k in enumerate([nv + 1, nv + 2, 33, 40, 48, 49, 64, 100, 257, 1500] * 3):
        k = max(k, nv + 1)
        pos[q:q + k] = pos[q]
        clump[q:q + k] = c
        q += k
    perm = rng.permutation(n)
    pos, clump = pos[perm], clump[perm]
    finder.configure(n, nvoisins=nv, nhop=min(16, nv))
    st = finder.run_stages(pos, np.full(n, 1.0 / n), last_stage=2, store_neighbours=nv)
    rows = st["neighbours"] - 1
    for c in range(clump.max() + 1):
        mem = np.nonzero(clump == c)[0]
        first = mem[:nv + 1]  # in index order
        for i in mem:
            assert np.array_equal(rows[i], first[first != i][:nv]), (c, len(mem), i)


@pytest.mark.parametrize("n,nmemb", [(20000, 20), (20000, 100), (120000, 20)])
def test_whole_finder(n, nmemb):
    # three clumps of coincident particles (infinite density) inside one dense
    # cloud, linked to its groups by finite saddles
    import oracle
    from ahop_b200 import finder
    rng = np.random.default_rng(3)
    pos = np.concatenate([rng.random((n - 9000, 3)) - 0.5, 0.01 * rng.normal(size=(9000, 3)) + 0.1])
    pos[:500] = [0.1, 0.1, 0.1]
    pos[500:540] = [0.112, 0.1, 0.1]
    pos[540:575] = [0.1, 0.115, 0.1]
    pos = pos[rng.permutation(n)]
    mass = np.full(n, 1.0 / n)
    finder.configure(n, nmembthresh=nmemb)
    got = finder.run(pos, mass)
    ref = oracle.run(pos, mass, oracle.default_params(n, nmembthresh=nmemb))
    assert got["ngroups"] == ref["ngroups"] and got["nnodes"] == ref["nnodes"]
    for f in ("density", "liste_parts", "integer_table", "real_table"):
        assert np.array_equal(got[f], ref[f]), f
