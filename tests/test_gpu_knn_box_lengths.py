"""Box lengths from where squared separations are subnormal floats to where they
near the largest: densities bit for bit the oracle's, and the FP32 scan only
where its margins hold (counters)."""
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


@pytest.mark.parametrize("box,per_lane", [(2.0 ** -45, False), (2.0 ** -30, False), (2.0 ** -26, True),
                                          (2.0 ** 20, True), (2.0 ** 49, True), (2.0 ** 52, False)])
def test_box_length(box, per_lane):
    import oracle
    from ahop_b200 import _lib, finder
    n = 100003
    rng = np.random.default_rng(21)
    pos = np.concatenate([1e-6 * rng.normal(size=(n // 2, 3)) + 0.2, rng.random((n - n // 2, 3)) - 0.5])
    pos = box * pos[rng.permutation(n)]  # a power of two: the same set at every length
    mass = np.full(n, 1.0 / n)
    finder.configure(n, box=box)
    lib = _lib.lib()
    lib.ahop_debug_set_task_profile(1)
    try:
        st = finder.run_stages(pos, mass, last_stage=2)
        out = (C.c_int64 * 30)()
        _lib.check(lib.ahop_debug_tree_stats(out, 30), "tree_stats")
    finally:
        lib.ahop_debug_set_task_profile(0)
    ref = oracle.run(pos, mass, oracle.default_params(n, box=box))
    assert np.array_equal(st["density"], ref["density"])
    assert (out[12] < out[8]) == per_lane, (out[12], out[8])
