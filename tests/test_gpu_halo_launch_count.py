"""Kernel launches reported by a property call: a replayed graph reports its own,
also when calls with other arguments came between."""
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


def test_launches_of_a_replay():
    import torch
    from ahop_b200 import halo_props
    rng = np.random.default_rng(8)
    off = np.array([0, 50, 400, 401])
    n = int(off[-1])
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    a = [t(off), t(0.01 * rng.normal(size=(n, 3))), t(rng.normal(size=(n, 3))), t(np.ones(n)), t(rng.random(n))]
    out = torch.zeros((3, halo_props.NF), dtype=torch.float64, device="cuda")

    def launches(epot):
        halo_props.compute_device(*a, out, 1.0, 0.0, epot=epot)
        return halo_props.timings()["kernel_launches"], halo_props.timings()["graph_replays"]

    first, r0 = launches(1)
    captured, r1 = launches(1)
    assert (captured, r0, r1) == (first, 0, 1)
    other, r = launches(0)
    assert other < first and r == 0
    again, r = launches(1)
    assert (again, r) == (first, 2)
