"""The FP32-compensated pair sum of a halo in parts of 128 rows (a call with a
few long work items) against the same halo in whole items (the same call with
enough other pairs), at the ends of rows, tiles and partner chunks."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,n,coincident", [
    (512, 10241, False), (512, 12000, False), (512, 16511, True), (512, 32768, False), (512, 33293, False),
    (256, 20481, False), (256, 33025, True), (256, 65900, False)])
def test_parts_equal_whole_items(rows, n, coincident):
    if not gpu_available():
        pytest.skip("no CUDA device")
    from ahop_b200 import build, halo_props
    build.build()
    rng = np.random.default_rng(n)
    longest = rows * min(n, 32768) - rows * rows // 2  # an item's own rows: each pair once
    big = int(np.sqrt(2.0 * 1.3 * 148 * 6 * rows * 32768))  # more pairs than every resident block's longest item
    pos = rng.normal(size=(n + big, 3))
    mass = rng.uniform(0.5, 1.5, n + big)
    if coincident:
        pos[n - 1] = pos[0]
        pos[n // 2] = pos[1]
    z = np.zeros_like(pos)

    def ep(off, epot=2):
        m = off[-1]
        r = halo_props.compute(np.asarray(off, np.int64), pos[:m], z[:m], mass[:m], mass[:m], 100.0, 0.0, 1.0, True,
                               epot=epot)
        return r, halo_props.timings()["items"]

    def whole_items(sizes):
        return sum(-(-(s - i) // 32768) for s in sizes for i in range(0, s, rows))

    halo_props.set_tiles([rows] * halo_props.BUCKETS)
    try:
        a, na = ep([0, n])
        b, nb = ep([0, n, n + big])
        f, _ = ep([0, n], epot=1)
    finally:
        halo_props.set_tiles(None)
    assert (na > whole_items([n])) == (longest >= 5 << 20) and nb == whole_items([n, big])
    a, b, f = a["ep32c"][0], b["ep32c"][0], f["ep64"][0]
    if coincident:
        # the per-pair recomputation covers the part, not the item: its rows'
        # sums have another order of additions, compensated in FP32 (2^-23 of a
        # row's sum, at most 512 of n rows)
        assert abs(a - b) <= 2.0 ** -23 * 512 / n * 4 * abs(b)
    else:
        # equal row sums; n FP64 terms of one sign in another order
        assert abs(a - b) <= n * 2.0 ** -53 * abs(b)
    assert abs(a - f) <= 1e-6 * abs(f)
