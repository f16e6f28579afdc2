"""The structure tree's ways of linking a task's groups give the oracle's tree:
component labels from the edge list in shared memory (narrow and wide blocks,
one CTA and clusters) and unions over the list in global memory (a wide task
that the shared array does not hold)."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    if not gpu_available():
        pytest.skip("no CUDA device")
    import oracle
    from ahop_b200 import build, synthetic
    build.build()
    ps = synthetic.small_box(60000, 12, seed=33, nmax=30000)
    return ps, oracle.run(ps.pos, ps.mass, oracle.default_params(ps.n))


@pytest.mark.parametrize("big,cap,ctas", [(512, 0, 4), (8, 0, 4), (8, 0, 1), (8, 16, 4), (8, 1, 1), (1, 64, 4)])
def test_linking_paths(case, big, cap, ctas):
    from ahop_b200 import _lib as L
    from ahop_b200 import finder
    ps, ref = case
    lib = L.lib()
    try:
        L.check(lib.ahop_debug_set_big_task(big))
        L.check(lib.ahop_debug_set_tree_par_cap(cap))
        L.check(lib.ahop_debug_set_tree_cluster(ctas))
        finder.configure(ps.n)
        out = finder.run(ps.pos, ps.mass)
    finally:
        L.check(lib.ahop_debug_set_big_task(512))
        L.check(lib.ahop_debug_set_tree_par_cap(0))
        L.check(lib.ahop_debug_set_tree_cluster(4))
    assert out["nnodes"] == ref["nnodes"] and out["nnodes"] > 50
    for f in ("integer_table", "real_table", "liste_parts", "density"):
        assert np.array_equal(out[f], ref[f]), f
