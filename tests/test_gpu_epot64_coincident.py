"""Coincident members in the FP64 potential: the sums leave them out, and only
the 256-partner tile that holds one is redone."""
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


def _case(sizes, dup, seed):
    rng = np.random.default_rng(seed)
    off = np.concatenate([[0], np.cumsum(sizes)])
    n = int(off[-1])
    pos = rng.normal(size=(n, 3)) * 0.01
    if dup:
        for h, k in enumerate(sizes):
            if k < 2:
                continue
            i, j = rng.choice(k, 2, replace=False)
            pos[off[h] + i] = pos[off[h] + j]
    return off, pos, rng.uniform(0.5, 1.5, n), rng.random(n)


def _ep(off, pos, mass, dens, rep=1):
    from ahop_b200 import halo_props
    best = np.inf
    for _ in range(rep):
        out = halo_props.compute(off, pos, np.zeros_like(pos), mass, dens, 1.0, 0.0, gravconst=1.0, epot=1)
        best = min(best, halo_props.timings()["epot64"])
    return out["ep64"], best


@pytest.mark.parametrize("sizes", [[2, 3, 33], [127, 128, 129, 255, 256, 257], [511, 512, 513, 700, 5000]])
def test_value(sizes):
    off, pos, mass, dens = _case(sizes, True, sum(sizes))
    got, _ = _ep(off, pos, mass, dens)
    for h in range(len(sizes)):
        p, m = pos[off[h]:off[h + 1]].astype(np.longdouble), mass[off[h]:off[h + 1]].astype(np.longdouble)
        c = p[np.argmax(dens[off[h]:off[h + 1]])]
        p = (p - c).astype(np.float64).astype(np.longdouble)  # separations from the rounded relative positions
        d = p[:, None] - p[None]
        r2 = (d * d).sum(2)
        with np.errstate(divide="ignore"):
            inv = np.where(r2 > 0, 1 / np.sqrt(r2), 0)
        pair = np.triu(inv * m[:, None] * m[None], 1)
        want = -pair.sum()
        # each term: its separations, square, root and product, ten roundings; the sum's own, one per term of a row
        assert abs(float(got[h] - want)) <= (10 + sizes[h]) * 2.0 ** -53 * float(pair.sum()), (h, sizes[h])


def test_cost():
    # 20 halos of 20,000 members: 40 rows of 4e9 pairs in all hold a spoiled
    # tile, which is one in 78 of a row's
    sizes = [20000] * 20
    plain = _ep(*_case(sizes, False, 1), rep=4)[1]
    dup = _ep(*_case(sizes, True, 1), rep=4)[1]
    assert dup <= 1.25 * plain, (dup, plain)
