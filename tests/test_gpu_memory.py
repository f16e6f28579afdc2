"""Device memory of the finder: a call takes what its own sizes need, whatever
smaller calls came before, and runs where just that is free."""
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


def _uniform(n):
    return np.random.default_rng(n).random((n, 3)) - 0.5


def _clustered(n):
    rng = np.random.default_rng(n)
    k = n // 300
    c = rng.random((k, 3)) - 0.5
    p = c[rng.integers(0, k, n)] + 0.004 * rng.normal(size=(n, 3))
    return np.mod(p + 0.5, 1.0) - 0.5


def _release():
    import torch
    from ahop_b200 import _lib
    _lib.check(_lib.lib().ahop_release_device_memory(), "release")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _run(pos):
    from ahop_b200 import finder
    n = len(pos)
    finder.configure(n)
    out = finder.run(pos, np.full(n, 1.0 / n))
    # the tables are views of the library's memory
    return {f: np.array(out[f]) for f in ("density", "liste_parts", "real_table", "integer_table")}


def _held(sizes, make=_uniform):
    """Bytes the finder holds after calls of these sizes on fresh buffers, and the last call's outputs."""
    import torch
    free = _release()
    for n in sizes:
        out = _run(make(n))
    torch.cuda.synchronize()
    return free - torch.cuda.mem_get_info()[0], out


# the driver hands out 2 MB pages: one more or less for each of the finder's 60 buffers
PAGES = 60 * (2 << 20)


def test_growth_takes_no_more():
    _held([1000])  # the context's own allocations
    alone = _held([10000000])[0]
    grown = _held([9000000, 10000000])[0]
    assert grown <= alone + PAGES, (grown, alone)


def test_growth_where_just_enough_is_free():
    import torch
    _held([1000])
    alone, want = _held([3300000], _clustered)
    free = _release()
    block = torch.empty(free - alone - PAGES, dtype=torch.uint8, device="cuda")
    try:
        _run(_clustered(2900000))
        got = _run(_clustered(3300000))
    finally:
        del block
        _release()
    assert len(want["real_table"]) > 100
    for f in want:
        assert np.array_equal(got[f], want[f]), f
