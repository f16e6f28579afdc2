"""The kNN's first bound, octave by octave: whatever octave the bound lies in
(31 below four squared box lengths, then 30 lower ones), no leaf is handed to
the query-by-query search for it."""
import numpy as np
import pytest

from conftest import gpu_available
from test_gpu_knn_scale import _counters

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not gpu_available():
        pytest.skip("no CUDA device")
    from ahop_b200 import build
    build.build()


@pytest.mark.parametrize("spacing", [1.6e-5, 2.0e-5, 2.5e-5, 3.2e-5, 4.0e-5])
def test_bound_octaves(spacing):
    # a uniform cube of 47^3 particles at this mean spacing: the 33rd distance
    # is about twice the spacing, so the five spacings cross the octaves of
    # d^2 about 2^-28, the lowest one of the first look in a unit box
    n = 47 ** 3
    rng = np.random.default_rng(3)
    pos = (rng.random((n, 3)) - 0.5) * (47 * spacing)
    _, c = _counters(pos)
    # 64 times the size: the same keys but for the few pairs that share a cell here
    _, base = _counters(64.0 * pos)
    assert abs(c["left"] - base["left"]) <= 10, (c, base)
