"""The profiling counter of bins laid lower or finer: a leaf with a tight clump
far below its first bound counts them, a uniform set hardly."""
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


def test_rebinned_counter():
    from ahop_b200 import _lib, finder
    n = 120000
    rng = np.random.default_rng(9)
    pos = rng.random((n, 3)) - 0.5
    # clumps of 150 around points that lie in otherwise empty leaves: the three
    # leaves of the first bound reach far beyond a clump's own extent
    k = 200
    c = rng.random((k, 3)) - 0.5
    pos[:150 * k] = (c[:, None] + 1e-4 * rng.normal(size=(k, 150, 3))).reshape(-1, 3)
    pos = np.mod(pos + 0.5, 1.0) - 0.5
    finder.configure(n)
    lib = _lib.lib()
    lib.ahop_debug_set_task_profile(1)
    try:
        finder.run_stages(pos, np.full(n, 1.0 / n), last_stage=2)
        out = (C.c_int64 * 30)()
        _lib.check(lib.ahop_debug_tree_stats(out, 30), "tree_stats")
    finally:
        lib.ahop_debug_set_task_profile(0)
    assert 0 < out[28] <= 6 * out[8]  # at most six times per query leaf
