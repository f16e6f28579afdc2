"""Finder stages against the oracle where their kernels change course: more
groups than the one-block forest takes, groups on both sides of 256 members,
node counts on both sides of the pairwise renumbering, and members whose
densities share a float key in long runs."""
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


def _many_halos():
    """Thousands of small clumps: many groups, many nodes of equal mass."""
    rng = np.random.default_rng(3)
    c = rng.random((6000, 3)) - 0.5
    k = rng.integers(40, 80, 6000)
    h = np.repeat(np.arange(6000), k)
    p = c[h] + 4e-4 * rng.normal(size=(len(h), 3))
    return np.concatenate([p, rng.random((60000, 3)) - 0.5])


def _lattice_clump():
    """A dense, very slightly irregular lattice: densities equal to a float."""
    rng = np.random.default_rng(4)
    g = np.stack(np.meshgrid(*[np.arange(14)] * 3, indexing="ij"), -1).reshape(-1, 3) * 1e-3
    p = g + 1e-12 * rng.random(g.shape)
    q = p + np.array([0.2, 0.1, 0.0])
    return np.concatenate([p, q[: len(q) // 2], 2e-3 * rng.normal(size=(3000, 3)) - 0.3, rng.random((9000, 3)) - 0.5])


@pytest.mark.parametrize("make", [_many_halos, _lattice_clump])
def test_stages_match_oracle(make):
    import oracle
    from ahop_b200 import finder
    pos = np.mod(make() + 0.5, 1.0) - 0.5
    pos = pos[np.random.default_rng(5).permutation(len(pos))]
    n = len(pos)
    mass = np.full(n, 1.0 / n)
    finder.configure(n)
    out = finder.run(pos, mass)
    ref = oracle.run(pos, mass, oracle.default_params(n))
    if make is _many_halos:
        assert ref["ngroups"] > 2048 and ref["nnodes"] > 4096
    assert out["ngroups"] == ref["ngroups"] and out["nnodes"] == ref["nnodes"]
    for f in ("density", "liste_parts", "integer_table", "real_table"):
        assert np.array_equal(out[f], ref[f]), f
