"""The FP64 direct sums over a halo's members against NumPy at the sizes where
the kernels change course: rows and partner tiles of 256 (two rows per thread),
partners split between items, coincident members, and the reciprocal square
root over its range."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 31, 33, 127, 128, 129, 255, 256, 257, 511, 512, 513, 769, 2050]


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not gpu_available():
        pytest.skip("no CUDA device")
    from ahop_b200 import build
    build.build()


def _ep64(off, pos, mass, box=100.0, periodic=True):
    from ahop_b200 import halo_props
    z = np.zeros_like(pos)
    return halo_props.compute(np.asarray(off, np.int64), pos, z, mass, mass, box, 0.0, 1.0, periodic, epot=1)["ep64"]


def _reference(pos, mass):
    """-sum_{i<j} m_i m_j / r_ij in extended precision, r = 0 left out."""
    d = pos[:, None].astype(np.longdouble) - pos[None]
    r2 = (d * d).sum(2)
    i, j = np.triu_indices(len(pos), 1)
    r2 = r2[i, j]
    return -float((mass[i] * mass[j] / np.sqrt(np.where(r2 > 0, r2, np.inf))).sum())


@pytest.mark.parametrize("coincident", [False, True])
def test_sums_at_tile_edges(coincident):
    rng = np.random.default_rng(7)
    off = np.concatenate([[0], np.cumsum(SIZES)])
    pos = rng.normal(size=(off[-1], 3))
    mass = rng.uniform(0.5, 1.5, off[-1])
    if coincident:
        for a, b in zip(off[:-1], off[1:]):
            for k in (0, (b - a) // 2):  # a neighbour in the same tile, the first member again at the end
                if a + k + 1 < b:
                    pos[a + k + 1] = pos[a + k]
            pos[b - 1] = pos[a]
    got = _ep64(off, pos, mass)
    for a, b, e in zip(off[:-1], off[1:], got):
        want = _reference(pos[a:b], mass[a:b])
        # positions relative to the centre are rounded once (2^-52 of ~5 over the
        # nearest separations), the sums' terms have one sign
        assert abs(e - want) <= 1e-12 * abs(want), (b - a, e, want)


def test_pairs_over_the_range_of_separations():
    # one member at the origin, the other on an axis at exactly representable
    # distances: two roundings of the product and the kernel's own 2 ulp
    rng = np.random.default_rng(8)
    d = 2.0 ** rng.uniform(-140, 140, 4000)
    pos = np.zeros((8000, 3))
    pos[1::2, 0] = d
    mass = np.tile([2.0, 1.0], 4000)  # the denser member, at the origin, is the centre
    got = _ep64(np.arange(0, 8001, 2), pos, mass, periodic=False)
    assert np.all(np.abs(got * d + 2.0) <= 2.0 * 4 * 2.0 ** -52)


@pytest.mark.parametrize("coincident", [False, True])
def test_gradient_at_tile_edges(coincident):
    import torch
    from ahop_b200 import autograd
    rng = np.random.default_rng(9)
    sizes = SIZES + [5000]  # partners of the largest go to ten items
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    pos = rng.normal(size=(off[-1], 3))
    mass = rng.uniform(0.5, 1.5, off[-1])
    if coincident:
        for a, b in zip(off[:-1], off[1:]):
            if b - a > 2:
                pos[b - 1] = pos[a]
                pos[a + (b - a) // 2] = pos[a]
    dev = torch.device("cuda:0")
    gh = rng.normal(size=len(sizes))
    p = torch.from_numpy(pos).to(dev).requires_grad_(True)
    e = autograd.HaloPotential.apply(p, torch.from_numpy(mass).to(dev), torch.from_numpy(off), 100.0, 1.0)
    e.backward(torch.from_numpy(gh).to(dev))
    grad = p.grad.cpu().numpy()
    for h, (a, b) in enumerate(zip(off[:-1], off[1:])):
        x, m = pos[a:b], mass[a:b]
        for i in rng.choice(b - a, min(b - a, 300), replace=False):
            d = x[i] - x
            r2 = (d * d).sum(1)
            w = m / np.where(r2 > 0, r2, np.inf) ** 1.5
            terms = gh[h] * m[i] * w[:, None] * d
            # each term within 1e-13 (separations of positions rounded once), n terms
            assert np.all(np.abs(grad[a + i] - terms.sum(0)) <= 1e-12 * np.abs(terms).sum(0) + 1e-300), (b - a, i)
