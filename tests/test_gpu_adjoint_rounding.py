"""Roundings of the density adjoint's pair term, on separations whose lengths
and ratios are exact: (a, b, c) units with an integer length e, a smoothing
length of a power of two units.  What is left are three roundings: the weight
times the kernel's derivative, over the distance, times the separation."""
import ctypes as C
from fractions import Fraction

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


def test_pair_term_roundings():
    import torch
    from ahop_b200 import _lib, autograd
    lib = autograd._bind()
    unit = 2.0 ** -12
    quads = [(a, b, c, int(round((a * a + b * b + c * c) ** 0.5))) for a in range(0, 40) for b in range(a, 40)
             for c in range(max(b, 1), 40)]
    quads = [q for q in quads if q[0] ** 2 + q[1] ** 2 + q[2] ** 2 == q[3] ** 2]
    cases = [(q, k) for q in quads for k in (16, 32, 64) if q[3] < 2 * k]  # e < 2 r: a term that is not zero
    m = len(cases)
    assert m > 100
    pos = np.zeros((3 * m, 3))
    nei = np.zeros((3 * m, 2), np.int32)
    g = np.zeros(3 * m)
    for t, ((a, b, c, e), k) in enumerate(cases):
        i = 3 * t
        pos[i] = 0.0
        pos[i + 1] = np.array([-a, b, -c]) * unit   # the neighbour
        pos[i + 2] = np.array([2 * k, 0, 0]) * unit  # the last one: r is k units
        nei[i:i + 3] = [[i + 1, i + 2], [i, i + 2], [i, i + 1]]
        g[i] = 1.0
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    p, w, n, gd = dev(pos), dev(np.ones(3 * m)), dev(nei), dev(g)
    out = torch.zeros((3 * m, 3), dtype=torch.float64, device="cuda")
    prm = autograd.AhopAdjParams(2, 0, 1.0, 1.0, 1.0)
    _lib.check(lib.ahop_density_adjoint(C.byref(prm), p.data_ptr(), w.data_ptr(), n.data_ptr(), 3 * m, gd.data_ptr(),
                                        out.data_ptr(), None), "density_adjoint")
    got = out.cpu().numpy()
    const = Fraction(1.0 / float(np.float32(3.141592654)))
    unit = Fraction(unit)
    bound = 3 * Fraction(2) ** -53 * (1 + Fraction(2) ** -50)
    worst = Fraction(0)
    for t, ((a, b, c, e), k) in enumerate(cases):
        u = Fraction(e, k)
        dw = -3 * u + Fraction(9, 4) * u * u if u <= 1 else -Fraction(3, 4) * (2 - u) ** 2
        coef = const * dw / (k * unit) ** 4 / (e * unit)
        # minus the neighbour's position: the separation the kernel forms is the particle's minus the neighbour's
        for ax, v in enumerate((-a, b, -c)):
            want = coef * v * unit
            x = Fraction(float(got[3 * t + 1, ax]))
            if want == 0:
                assert x == 0
            else:
                worst = max(worst, abs(abs(x) - abs(want)) / abs(want))
                assert (x > 0) == (want > 0)
    assert worst <= bound, float(worst * 2 ** 53)
