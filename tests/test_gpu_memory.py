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


def test_bytes_per_particle():
    # without groups, by array: inputs 32, sort keys, permutations, hop targets
    # and roots 32, sorted x, y, z, m 32, index and rank 8, boxes 80 per 31,
    # neighbours 64, density in both orders 16, group, peak flag, members and
    # node ids 16, the radix sort's second copy of keys and values 12; from 8.4M
    # particles on the kNN's collected slots are no larger (1.65 GB)
    _held([1000])
    small = _held([9000000])[0]
    large = _held([18000000])[0]
    assert large - small <= 9000000 * 214.6 + PAGES, (large - small) / 9e6
    assert large <= 18000000 * 214.6 + 1.66e9 + PAGES, large


def test_groups_view_needs_its_stage():
    from ahop_b200 import _lib, finder
    pos = _uniform(5000)
    finder.configure(5000)
    finder.run_stages(pos, np.full(5000, 2e-4), last_stage=2)
    hop = np.zeros(5000, np.int32)
    assert _lib.lib().ahop_debug_groups(hop.ctypes.data, hop.ctypes.data, None) == 4  # ESTATE


def test_growth_where_just_enough_is_free():
    import torch
    _held([1000])
    alone, want = _held([3300000], _clustered)
    free = _release()
    try:
        block = torch.empty(free - alone - PAGES, dtype=torch.uint8, device="cuda")
    except torch.OutOfMemoryError:
        pytest.skip("another process took device memory meanwhile")
    try:
        _run(_clustered(2900000))
        got = _run(_clustered(3300000))
    finally:
        del block
        _release()
    assert len(want["real_table"]) > 100
    for f in want:
        assert np.array_equal(got[f], want[f]), f
