"""The kNN's leaves at scales far below the box: a clump 1e-5 of the box across
is searched leaf by leaf as the same clump is at a thousand times the size
(counters of the profiled kernels), with the oracle's densities."""
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


def _counters(pos):
    from ahop_b200 import _lib, finder
    n = len(pos)
    finder.configure(n)
    lib = _lib.lib()
    lib.ahop_debug_set_task_profile(1)
    try:
        st = finder.run_stages(pos, np.full(n, 1.0 / n), last_stage=2)
        out = (C.c_int64 * 30)()
        _lib.check(lib.ahop_debug_tree_stats(out, 30), "tree_stats")
    finally:
        lib.ahop_debug_set_task_profile(0)
    return st, dict(leaves=out[8], candidates=out[9], left=out[12], queries_left=out[18])


def test_small_clump_leaves():
    import oracle
    n = 131072
    rng = np.random.default_rng(5)
    shape = rng.normal(size=(n - 64, 3))
    rest = rng.random((64, 3)) - 0.5
    perm = rng.permutation(n)
    large = np.concatenate([0.01 * shape + 0.1, rest])[perm]
    small = np.concatenate([1e-5 * shape + 0.1, rest])[perm]
    _, a = _counters(large)
    st, b = _counters(small)
    assert a["leaves"] == b["leaves"] == n // 32
    # a key's cell is 2^-21 of the box, 1/21 of this clump's sigma: the leaves
    # are the larger clump's up to where cell walls fall
    assert b["left"] <= 2 * a["left"] + 0.01 * b["leaves"], (a, b)
    assert b["candidates"] <= 1.5 * a["candidates"], (a, b)
    ref = oracle.run(small, np.full(n, 1.0 / n), oracle.default_params(n))
    assert np.array_equal(st["density"], ref["density"])
