"""Measured cases of the halo finder and the stages next to it.

A case is one call (or one forward + backward pass) through an entry point that a program of this
package's users calls: the drop-in finder on host arrays, the finder on device arrays, a whole snapshot,
the batched halo properties, the differentiable density and potential, and the RAMSES part-file reader.

Particles are the boxes of ahop_b200.synthetic drawn on the GPU: NFW halos (concentration 10, virial
radius 0.01 (n / 1000)^(1/3) of the box) with 0-4 subhalos of 2-10 % each over a uniform background,
particle order shuffled as in a snapshot.  Halo sizes are the quantiles of dN/dn ~ n^-1.9, so that a
case costs the same whatever its seed; positions, velocities and order come from the seed.

listed() holds the sizes of the repository's tests and benchmark and generic ones between them;
draw(rng) gives more of the same ranges; prepare(case, seed) makes what a program has in hand before
the call; run(state) is one pass and returns its outputs; exact(case, seed) is the same in plain
64-bit torch; work(case) is what a pass cannot do without.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "halomaker-python_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ctypes  # noqa: E402

from ahop_b200 import _lib as lib  # noqa: E402
from ahop_b200 import autograd, finder, halo_props, pipeline, ramses  # noqa: E402
from compute_adaptahop import neikdtree  # noqa: E402

DEV = "cuda"
TREE = ("mother", "first_sister", "first_daughter", "level", "ids", "offsets")
NFW_C = 10.0
HUB = 70.0
G = 430.1
SCALE_L, SCALE_T = 3.0e24, 4.5e17  # cm and s: the units of a RAMSES info file


def listed():
    return [
        # one small zoom region or a test box through the drop-in module: all latency and launches
        dict(name="finder_5k", kind="finder", n=5_003, nhalo=12, nmax=1_000, nv=32, nhop=16, box=1.0, stars=0.0),
        # a mid-size box with fewer neighbours, in a 100-unit box, as the reference's driver passes it
        dict(name="finder_70k_nv20", kind="finder", n=70_001, nhalo=80, nmax=8_000, nv=20, nhop=10, box=100.0,
             stars=0.0),
        # the 262,144-particle configuration of the benchmark file through the drop-in module
        dict(name="finder_262k", kind="finder", n=262_144, nhalo=300, nmax=20_000, nv=32, nhop=16, box=1.0,
             stars=0.0),
        # dark matter with 15 % stars in the halo cores (family = all), ragged size
        dict(name="finder_2m_stars", kind="finder", n=2_000_003, nhalo=2_000, nmax=50_000, nv=32, nhop=16, box=1.0,
             stars=0.15),
        # the benchmark's 256^3 box on device arrays, as the snapshot pipeline calls the finder
        dict(name="finder_256cubed", kind="finder_device", n=16_777_216, nhalo=19_200, nmax=2_000_000, nv=32,
             nhop=16, box=1.0, stars=0.0),
        # a whole snapshot: finder, halo selection, member gather, properties, virial step
        dict(name="snapshot_1m", kind="snapshot", n=1_000_000, nhalo=1_000, nmax=30_000, nv=32, nhop=16, box=1.0,
             stars=0.15),
        # halo properties with both forms of the potential on a small catalogue
        dict(name="props_200_both", kind="props", nhalo=200, nmin=20, nmax=3_000, epot=3),
        # FP64 direct sum, the form compared with the reference
        dict(name="props_2000_fp64", kind="props", nhalo=2_000, nmin=20, nmax=200_000, epot=1),
        # the benchmark's 20,000-halo catalogue, FP32-compensated potential
        dict(name="props_20000_fp32c", kind="props", nhalo=20_000, nmin=20, nmax=2_000_000, epot=2),
        # density of a 2M-particle box with fixed neighbour lists, forward and backward
        dict(name="density_grad_2m", kind="density", n=2_097_152, nhalo=2_000, nmax=50_000, nv=32),
        # potential of every halo of a catalogue, forward and backward (forces)
        dict(name="potential_grad_500", kind="potential", nhalo=500, nmin=20, nmax=30_000),
        # RAMSES part files (Ra4, dark matter and stars) to device arrays
        dict(name="reader_1m", kind="reader", n=1_000_003, nfiles=8, version=4, stars=0.15),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["finder", "finder", "finder", "finder_device", "finder_device", "snapshot", "props", "props",
                       "density", "potential", "reader"])
    if kind in ("finder", "finder_device"):
        n = _logint(rng, 3_000, 2_500_000 if kind == "finder" else 16_777_216)
        nv = rng.choice([16, 20, 24, 32, 32, 32])
        return dict(kind=kind, n=n, nhalo=max(4, n // rng.randint(700, 1_100)),
                    nmax=max(200, min(2_000_000, n // rng.randint(8, 40))), nv=nv, nhop=rng.randint(8, 16),
                    box=rng.choice([1.0, 1.0, 100.0]), stars=rng.choice([0.0, 0.0, 0.15]))
    if kind == "snapshot":
        n = _logint(rng, 20_000, 2_000_000)
        return dict(kind=kind, n=n, nhalo=max(8, n // rng.randint(700, 1_100)), nmax=max(400, n // rng.randint(20, 60)),
                    nv=32, nhop=16, box=1.0, stars=rng.choice([0.0, 0.15]))
    if kind == "props":
        nhalo = _logint(rng, 50, 20_000)
        return dict(kind=kind, nhalo=nhalo, nmin=20, nmax=_logint(rng, 500, 150_000), epot=rng.choice([1, 2, 3]))
    if kind == "density":
        n = _logint(rng, 10_000, 2_097_152)
        return dict(kind=kind, n=n, nhalo=max(4, n // 1_000), nmax=max(300, n // 30), nv=rng.choice([16, 24, 32]))
    if kind == "potential":
        return dict(kind=kind, nhalo=_logint(rng, 20, 2_000), nmin=20, nmax=_logint(rng, 500, 50_000))
    return dict(kind="reader", n=_logint(rng, 20_000, 2_000_000), nfiles=rng.choice([2, 8, 16, 32]),
                version=rng.choice([3, 4]), stars=rng.choice([0.0, 0.15]))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1_000_003 + 17)


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)


def _counts(nhalo, nmin, nmax, slope=-1.9):
    """Halo sizes: the quantiles of dN/dn ~ n^slope on [nmin, nmax], largest first."""
    a = slope + 1.0
    u = (np.arange(nhalo) + 0.5) / nhalo
    lo, hi = float(nmin) ** a, float(nmax) ** a
    return np.floor((lo + u * (hi - lo)) ** (1.0 / a)).astype(np.int64)[::-1].copy()


def _nfw_radius(g, n):
    """Radii in units of the virial radius, by the inverse of the NFW enclosed mass."""
    x = torch.linspace(0.0, 1.0, 4097, device=DEV, dtype=torch.float64)
    m = torch.log1p(NFW_C * x) - NFW_C * x / (1.0 + NFW_C * x)
    cdf = m / m[-1]
    u = _rand(g, n)
    k = torch.searchsorted(cdf, u).clamp(1, 4096)
    t = (u - cdf[k - 1]) / (cdf[k] - cdf[k - 1])
    return x[k - 1] + t * (x[k] - x[k - 1])


def _isotropic(g, n):
    v = _randn(g, n, 3)
    return v / (v.norm(dim=1, keepdim=True) + 1e-300)


def _wrapped(p, box):
    """Into [-box/2, box/2)."""
    p = torch.remainder(p, box)
    p = torch.where(p >= box, torch.zeros_like(p), p) - 0.5 * box
    return torch.where(p >= 0.5 * box, torch.full_like(p, -0.5 * box), p)


def _box(case, seed):
    """pos (n,3), vel (n,3), mass (n,) and the dark-matter count (None: all) of a clustered box, on the GPU."""
    g = _gen(seed)
    n, box, stars = case["n"], case.get("box", 1.0), case.get("stars", 0.0)
    counts = _counts(case["nhalo"], 20, case["nmax"])
    counts = np.maximum(20, np.floor(counts * (0.6 * n / counts.sum()))).astype(np.int64)
    while counts.sum() > n:  # tiny boxes: the floor of 20 may overshoot
        counts = counts[:-1]
    cnt = torch.from_numpy(counts).to(DEV)
    nh = len(counts)
    centre = _rand(g, nh, 3) * box
    rvir = 0.01 * box * (cnt.double() / 1000.0) ** (1.0 / 3.0)
    # subhalos: up to four per halo, each 2-10 % of its particles, 0.3-0.8 r_vir from its centre
    nsub = torch.floor(_rand(g, nh) * 5.0)
    frac = 0.02 + 0.08 * _rand(g, nh, 4)
    slot = torch.arange(4, device=DEV)
    sub = torch.where(slot[None, :] < nsub[:, None], torch.floor(cnt.double()[:, None] * frac), 0.0).long()
    sub[sub < 2] = 0
    sub_c = centre[:, None, :] + (0.3 + 0.5 * _rand(g, nh, 4))[..., None] * rvir[:, None, None] * _isotropic(
        g, nh * 4).reshape(nh, 4, 3)
    blob_n = torch.cat([(cnt - sub.sum(1))[:, None], sub], 1)
    blob_c = torch.cat([centre[:, None, :], sub_c], 1).reshape(-1, 3)
    blob_r = 0.01 * box * (blob_n.double() / 1000.0) ** (1.0 / 3.0)
    blob_r[:, 0] = rvir
    blob_r, blob_h = blob_r.reshape(-1), torch.arange(nh, device=DEV).repeat_interleave(5)
    of = torch.repeat_interleave(torch.arange(nh * 5, device=DEV), blob_n.reshape(-1))
    nhp = of.numel()
    hid = blob_h[of]
    pos = torch.empty((n, 3), dtype=torch.float64, device=DEV)
    vel = torch.empty((n, 3), dtype=torch.float64, device=DEV)
    pos[:nhp] = blob_c[of] + (_nfw_radius(g, nhp) * blob_r[of])[:, None] * _isotropic(g, nhp)
    sig = 100.0 * (cnt.double() / 1000.0) ** (1.0 / 3.0)
    vel[:nhp] = sig[hid][:, None] * _randn(g, nhp, 3) + (300.0 * _randn(g, nh, 3))[hid]
    mass = torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV)
    is_star = torch.zeros(n, dtype=torch.bool, device=DEV)
    if stars > 0.0:  # Plummer cores of half-mass radius 0.05 r_vir, particles of a tenth of the mass
        is_star[:nhp] = _rand(g, nhp) < stars
        k = is_star[:nhp].nonzero().squeeze(1)
        a = 0.05 * rvir[hid[k]] / 1.305
        rs = torch.minimum(a / torch.sqrt(_rand(g, k.numel()) ** (-2.0 / 3.0) - 1.0), rvir[hid[k]])
        pos[k] = centre[hid[k]] + rs[:, None] * _isotropic(g, k.numel())
        mass[is_star] *= 0.1
        mass /= mass.sum()
    pos[nhp:] = _rand(g, n - nhp, 3) * box
    vel[nhp:] = 30.0 * _randn(g, n - nhp, 3)
    pos = _wrapped(pos, box)
    perm = torch.randperm(n, generator=g, device=DEV)
    ndm = None
    if stars > 0.0:  # dark matter first, then stars, as the reader lays out family = all
        perm = perm[torch.argsort(is_star[perm].to(torch.int8), stable=True)]
        ndm = int(n - int(is_star.sum()))
    return pos[perm].contiguous(), vel[perm].contiguous(), mass[perm].contiguous(), ndm


CAT_BOX = 100.0


def _catalogue(case, seed):
    """Offsets (host), pos, vel, mass, density of a catalogue of grouped halos in a 100-unit box."""
    g = _gen(seed)
    counts = _counts(case["nhalo"], case["nmin"], case["nmax"])
    order = torch.randperm(len(counts), generator=g, device=DEV).cpu().numpy()
    counts = counts[order]
    off = np.zeros(len(counts) + 1, np.int64)
    np.cumsum(counts, out=off[1:])
    cnt = torch.from_numpy(counts).to(DEV)
    hid = torch.repeat_interleave(torch.arange(len(counts), device=DEV), cnt)
    n = int(off[-1])
    rvir = 0.01 * CAT_BOX * (cnt.double() / 1000.0) ** (1.0 / 3.0)
    x = _nfw_radius(g, n)
    pos = ((_rand(g, len(counts), 3) - 0.5) * CAT_BOX)[hid] + (x * rvir[hid])[:, None] * _isotropic(g, n)
    pos = _wrapped(pos + 0.5 * CAT_BOX, CAT_BOX).contiguous()
    sig = 100.0 * (cnt.double() / 1000.0) ** (1.0 / 3.0)
    vel = (sig[hid][:, None] * _randn(g, n, 3) + (300.0 * _randn(g, len(counts), 3))[hid]).contiguous()
    xm = torch.clamp(x, min=1e-4)
    dens = 1.0 / (xm * (1.0 + 10.0 * xm) ** 2) * (1.0 + 1e-3 * _rand(g, n))
    mass = 0.5 + _rand(g, n)
    return off, pos, vel, mass, dens


def _part_files(case, seed):
    """Part files in the RAMSES layout in a temporary directory: the directory (removed with the object),
    the paths, and the table (x, v, m and the dense row of every particle) they hold."""
    rng = np.random.Generator(np.random.PCG64(seed))
    n, nfiles, version = case["n"], case["nfiles"], case["version"]
    nstar = int(case["stars"] * n)
    star = np.zeros(n, bool)
    star[rng.permutation(n)[:nstar]] = True
    ids = np.empty(n, np.int32)
    ids[~star] = rng.permutation(n - nstar) + 1
    ids[star] = rng.permutation(nstar) + 1
    row = ids.astype(np.int64) - 1
    row[star] += n - nstar
    x, v = rng.random((n, 3)), rng.normal(scale=0.05, size=(n, 3))
    m = np.where(star, 1e-7, 1e-6) * rng.uniform(0.9, 1.1, n)
    birth = np.where(star, -rng.uniform(0.1, 5.0, n), 0.0)
    fam = np.where(star, 2, 1).astype(np.int8)
    bounds = np.concatenate([[0], np.sort(rng.integers(0, n + 1, nfiles - 1)), [n]])
    hold = tempfile.TemporaryDirectory(prefix="parts_")
    paths = []
    for c in range(nfiles):
        a, b = int(bounds[c]), int(bounds[c + 1])
        k = b - a
        recs = [np.array([nfiles], np.int32), np.array([3], np.int32), np.array([k], np.int32),
                np.arange(4, dtype=np.int32), np.array([nstar], np.int32), np.array([1.5e-3]), np.array([0.0]),
                np.array([0], np.int32)]
        recs += [x[a:b, d] for d in range(3)] + [v[a:b, d] for d in range(3)]
        recs += [m[a:b], ids[a:b], np.full(k, 9, np.int32)]
        if version == 4:
            recs += [fam[a:b], np.zeros(k, np.int8)]
        if nstar > 0:
            recs += [birth[a:b], np.zeros(k)]
        path = os.path.join(hold.name, "part_00001.out%05d" % (c + 1))
        with open(path, "wb") as f:
            for r in recs:
                r = np.ascontiguousarray(r)
                size = np.array([r.nbytes], np.uint32).tobytes()
                f.write(size)
                f.write(r.tobytes())
                f.write(size)
        paths.append(path)
    return hold, paths, dict(x=x, v=v, m=m, row=row)


def _configure(s):
    c = s["case"]
    finder.configure(c["n"], box=c["box"], nvoisins=c["nv"], nhop=c["nhop"])


class _Array:
    """Device memory of the library as an array that torch can view."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=3)


def _view(ptr, shape, typestr):
    if not ptr or 0 in shape:
        return torch.empty(shape, dtype=torch.float64 if typestr == "<f8" else torch.int32, device=DEV)
    return torch.as_tensor(_Array(int(ptr), shape, typestr), device=DEV)


def _rows(case):
    """Rows of the arrays that keep a snapshot's structure tables (their number depends on the particles)."""
    return 8 * case["nhalo"] + 64


def _keep(buf, table):
    """A structure table copied into the program's own array, the rest of it cleared."""
    buf[:len(table)] = table
    buf[len(table):] = 0
    return buf


# ------------------------------------------------------------------ the cases
def prepare(case, seed):
    k = case["kind"]
    s = dict(case=case)
    if k in ("finder", "snapshot"):
        pos, vel, mass, ndm = _box(case, seed)
        s.update(pos=pos.cpu().numpy(), mass=mass.cpu().numpy(), ndm=ndm)
        rows = _rows(case)
        if k == "snapshot":
            s.update(vel=vel.cpu().numpy(), props=np.zeros((rows, halo_props.NF)),
                     virial=np.zeros((rows, halo_props.NV)))
            s.update({f: np.zeros(rows, np.int32) for f in TREE})
        else:
            s.update(real=np.zeros((rows, 8)), integer=np.zeros((rows, 6), np.int32))
    elif k == "finder_device":
        pos, _, mass, _ = _box(case, seed)
        s.update(pos=pos, mass=mass, real=torch.zeros((_rows(case), 8), dtype=torch.float64, device=DEV),
                 integer=torch.zeros((_rows(case), 6), dtype=torch.int32, device=DEV))
    elif k == "props":
        off, pos, vel, mass, dens = _catalogue(case, seed)
        s.update(off=torch.from_numpy(off).to(DEV), pos=pos, vel=vel, mass=mass, dens=dens,
                 out=torch.zeros((case["nhalo"], halo_props.NF), dtype=torch.float64, device=DEV))
    elif k == "density":
        pos, _, mass, _ = _box(case, seed)
        finder.configure(case["n"], nvoisins=case["nv"], nhop=min(16, case["nv"]))
        st = finder.run_stages(pos.cpu().numpy(), mass.cpu().numpy(), last_stage=2, store_neighbours=case["nv"])
        nei = torch.from_numpy(np.ascontiguousarray(st["neighbours"] - 1, np.int32)).to(DEV)
        s.update(pos=pos, mass=mass, nei=nei, g=_randn(_gen(seed + 1), case["n"]))
    elif k == "potential":
        off, pos, _, mass, _ = _catalogue(case, seed)
        s.update(off=torch.from_numpy(off), pos=pos, mass=mass, g=_randn(_gen(seed + 1), case["nhalo"]))
    else:
        hold, paths, _ = _part_files(case, seed)
        s.update(hold=hold, paths=paths)
    if k in ("props", "snapshot"):
        halo_props.set_tiles([128, 128, 256, 512, 512])  # pinned: the same FP32 bits in every process
    torch.cuda.synchronize()
    return s


def run(s):
    c = s["case"]
    k = c["kind"]
    if k == "finder":
        _configure(s)
        neikdtree.compute_adaptahop(s["pos"].T, s["mass"])
        # the reference's driver copies the tables out before it closes the module
        return dict(density=neikdtree.density, liste_parts=neikdtree.liste_parts,
                    real_table=_keep(s["real"], neikdtree.real_table.T),
                    integer_table=_keep(s["integer"], neikdtree.integer_table.T))
    if k == "finder_device":
        _configure(s)
        L = lib.lib()
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        lib.check(L.ahop_compute_adaptahop_device(s["pos"].data_ptr(), s["mass"].data_ptr(), c["n"], stream))
        o = lib.AhopOutputs()
        lib.check(L.ahop_get_device_outputs(ctypes.byref(o)))
        nn = int(o.nnodes)
        return dict(density=_view(o.density, (c["n"],), "<f8"), liste_parts=_view(o.liste_parts, (c["n"],), "<i4"),
                    real_table=_keep(s["real"], _view(o.real_table, (nn, 8), "<f8")),
                    integer_table=_keep(s["integer"], _view(o.integer_table, (nn, 6), "<i4")))
    if k == "snapshot":
        r = pipeline.run_snapshot(s["pos"], s["vel"], s["mass"], box=c["box"], hub=HUB,
                                  finder_params=dict(nvoisins=c["nv"], nhop=c["nhop"]), particle_views=True,
                                  ndm=s["ndm"])
        return dict({f: _keep(s[f], r[f]) for f in TREE + ("props", "virial")}, whereIam_parts=r["whereIam_parts"],
                    pids_groupsorted=r["pids_groupsorted"])
    if k == "props":
        halo_props.compute_device(s["off"], s["pos"], s["vel"], s["mass"], s["dens"], s["out"], CAT_BOX, HUB, G,
                                  epot=c["epot"], stream=torch.cuda.current_stream())
        return s["out"].unbind(1)
    if k == "density":
        p = s["pos"].detach().requires_grad_(True)
        rho = autograd.SPHDensity.apply(p, s["mass"], s["nei"], 1.0)
        rho.backward(s["g"])
        return dict(density=rho, grad=p.grad)
    if k == "potential":
        p = s["pos"].detach().requires_grad_(True)
        e = autograd.HaloPotential.apply(p, s["mass"], s["off"], CAT_BOX, G)
        e.backward(s["g"])
        return dict(energy=e, grad=p.grad)
    r = ramses.read_parts(s["paths"], c["version"], "all", SCALE_L, SCALE_T)
    return dict(pos=r["pos"], vel=r["vel"], mass=r["mass"], ndm=r["ndm"], nstar=r["nstar"])


def _pairs(case):
    n = _counts(case["nhalo"], case["nmin"], case["nmax"]).astype(np.float64)
    return float(n.sum()), float((n * (n - 1) / 2).sum())


def work(case):
    """Inputs read once, outputs written once; operations of the pairs and neighbours that define the result."""
    k = case["kind"]
    if k in ("finder", "finder_device"):
        # positions, masses in; density, node ids out; distance (9) and spline (10) per neighbour
        return dict(bytes=case["n"] * (32 + 12), flops=case["n"] * case["nv"] * 19.0)
    if k == "snapshot":
        return dict(bytes=case["n"] * (56 + 8), flops=case["n"] * case["nv"] * 19.0)
    if k == "props":
        n, pairs = _pairs(case)
        forms = (case["epot"] & 1) + (case["epot"] >> 1)
        return dict(bytes=n * 64 + case["nhalo"] * 8 * halo_props.NF, flops=n * 80 + forms * pairs * 20.0)
    if k == "density":
        return dict(bytes=case["n"] * (2 * (24 + 8 + 4 * case["nv"]) + 8 + 8 + 24), flops=case["n"] * case["nv"] * 60.0)
    if k == "potential":
        n, pairs = _pairs(case)
        return dict(bytes=n * (24 + 8 + 24), flops=pairs * (20.0 + 30.0))
    per = 56 + 4 + (1 if case["version"] == 4 else 0) + (8 if case["version"] == 3 and case["stars"] > 0 else 0)
    return dict(bytes=case["n"] * (per + 56), flops=case["n"] * 9.0)


# ------------------------------------------------------------------ the same in plain 64-bit torch
PI_F = float(np.float32(3.141592654))  # the reference's single-precision literal is part of the definition


def _spline(u):
    return torch.where(u <= 1.0, 1.0 - 1.5 * u * u + 0.75 * u * u * u,
                       torch.where(u <= 2.0, 0.25 * (2.0 - u) ** 3, torch.zeros_like(u)))


def _density_of(d, m, m_self, volume):
    """d (rows, nv) ascending distances, m their masses: the density of the nv - 1 nearest."""
    r = 0.5 * d[:, -1]
    s = (m[:, :-1] * _spline(d[:, :-1] / r[:, None])).sum(1) + m_self
    return volume * s / (PI_F * r ** 3)


def _exact_density(pos, mass, nv, box):
    n = pos.shape[0]
    out = torch.empty(n, dtype=torch.float64, device=DEV)
    step = max(1, int(2.5e8) // n)
    for a in range(0, n, step):
        q = pos[a:a + step]
        d2 = torch.zeros((q.shape[0], n), dtype=torch.float64, device=DEV)
        for k in range(3):
            dx = (q[:, k:k + 1] - pos[None, :, k]).abs_()
            dx = torch.minimum(dx, box - dx)
            d2.addcmul_(dx, dx)
        i = torch.arange(q.shape[0], device=DEV)
        d2[i, a + i] = math.inf
        v, j = torch.topk(d2, nv, dim=1, largest=False, sorted=True)
        out[a:a + step] = _density_of(v.sqrt(), mass[j], mass[a:a + step], box ** 3)
    return out


def _wrap(d, box):
    d = torch.where(d > 0.5 * box, d - box, d)
    return torch.where(d < -0.5 * box, d + box, d)


def _pair_sums(off, rel, mass, grad=None):
    """sum_{i<j} m_i m_j / r_ij of every halo; with grad, minus its gradient with respect to rel goes there."""
    out = torch.zeros(len(off) - 1, dtype=torch.float64, device=DEV)
    for h in range(len(off) - 1):
        a, b = int(off[h]), int(off[h + 1])
        x, m = rel[a:b], mass[a:b]
        step = max(1, int(1e8) // max(1, b - a))
        for i in range(0, b - a, step):
            e = min(i + step, b - a)
            d = [x[i:e, k:k + 1] - x[None, :, k] for k in range(3)]
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
            w = torch.where(r2 > 0.0, r2, torch.full_like(r2, math.inf)).rsqrt_()
            out[h] += 0.5 * (m[i:e] * (w @ m)).sum()
            if grad is not None:
                w = w * w * w * m[None, :]
                for k in range(3):
                    grad[a + i:a + e, k] = m[i:e] * (w * d[k]).sum(1)
    return out


def _exact_props(case, seed):
    off, pos, vel, mass, dens = _catalogue(case, seed)
    nh, L = case["nhalo"], CAT_BOX
    cnt = torch.from_numpy(np.diff(off)).to(DEV)
    start = torch.from_numpy(off[:-1]).to(DEV)
    hid = torch.repeat_interleave(torch.arange(nh, device=DEV), cnt)
    tot = lambda v: torch.zeros(nh, dtype=torch.float64, device=DEV).index_add_(0, hid, v)
    order = torch.argsort(dens, descending=True, stable=True)
    order = order[torch.argsort(hid[order], stable=True)]
    ic = order[start]
    c = pos[ic]
    mt = tot(mass)
    vb = torch.stack([tot(mass * vel[:, k]) / mt for k in range(3)], 1)
    dr, u = _wrap(pos - c[hid], L), vel - vb[hid]
    p = mass[:, None] * u
    am = [tot(dr[:, (k + 1) % 3] * p[:, (k + 2) % 3] - dr[:, (k + 2) % 3] * p[:, (k + 1) % 3]) for k in range(3)]
    inertia = {(i, j): tot(mass * dr[:, i] * dr[:, j]) for i in range(3) for j in range(i, 3)}
    mat = torch.stack([inertia[min(i, j), max(i, j)] for i in range(3) for j in range(3)], 1).reshape(nh, 3, 3)
    ax = torch.sqrt(torch.linalg.eigvalsh(mat) / mt[:, None])
    t = u + dr * HUB
    ek = 0.5 * tot(mass * (t * t).sum(1))
    sig2 = tot(mass * (u * u).sum(1))
    res = dict(m=mt, px=c[:, 0], py=c[:, 1], pz=c[:, 2], vx=vb[:, 0], vy=vb[:, 1], vz=vb[:, 2], Lx=am[0], Ly=am[1],
               Lz=am[2], ek=ek, sigma=torch.sqrt(sig2 / mt), sha=ax[:, 0], shb=ax[:, 1], shc=ax[:, 2],
               icenter=(ic - start).double(), ndm=cnt.double(), mdm=mt, sigma_dm=torch.sqrt(sig2 / mt))
    r2 = torch.zeros(nh, dtype=torch.float64, device=DEV)
    res["r"] = torch.sqrt(r2.scatter_reduce_(0, hid, (dr * dr).sum(1), "amax"))
    for (i, j), v in inertia.items():
        res["I" + "xyz"[i] + "xyz"[j]] = v
    if _pairs(case)[1] < 2e11:
        ep = -G * _pair_sums(off, dr, mass)
        spin = torch.sqrt(am[0] ** 2 + am[1] ** 2 + am[2] ** 2) * torch.sqrt((ek + ep).abs()) / mt ** 2.5 / G
        if case["epot"] & 1:
            res.update(ep64=ep, spin64=spin)
        if case["epot"] & 2:
            res.update(ep32c=ep, spin32c=spin)
    return tuple(res.get(f) for f in halo_props.FIELDS)


def exact(case, seed):
    k = case["kind"]
    if k in ("finder", "finder_device"):
        if case["n"] > 300_000:  # all pairs: over 20 s
            return None
        pos, _, mass, _ = _box(case, seed)
        return dict(density=_exact_density(pos, mass, case["nv"], case["box"]), liste_parts=None, real_table=None,
                    integer_table=None)
    if k == "snapshot":
        return None
    if k == "props":
        return _exact_props(case, seed)
    if k == "density":
        s = prepare(case, seed)
        p = s["pos"].detach().requires_grad_(True)
        nei = s["nei"].long()
        d = p[:, None, :] - p[nei]
        d = torch.where(d > 0.5, d - 1.0, torch.where(d < -0.5, d + 1.0, d))
        rho = _density_of(d.square().sum(2).sqrt(), s["mass"][nei], s["mass"], 1.0)
        rho.backward(s["g"])
        return dict(density=rho.detach(), grad=p.grad)
    if k == "potential":
        off, pos, _, mass, _ = _catalogue(case, seed)
        cnt = torch.from_numpy(np.diff(off)).to(DEV)
        hid = torch.repeat_interleave(torch.arange(case["nhalo"], device=DEV), cnt)
        rel = _wrap(pos - pos[torch.from_numpy(off[:-1]).to(DEV)][hid], CAT_BOX)
        grad = torch.empty_like(pos)
        e = -G * _pair_sums(off, rel, mass, grad)
        gh = _randn(_gen(seed + 1), case["nhalo"])
        return dict(energy=e, grad=grad * (G * gh[hid])[:, None])
    _, _, t = _part_files(case, seed)
    n = case["n"]
    pos, vel, mass = np.empty((n, 3)), np.empty((n, 3)), np.empty(n)
    pos[t["row"]] = t["x"] - 0.5
    vel[t["row"]] = t["v"] * SCALE_L / SCALE_T * 1e-5
    mass[t["row"]] = t["m"]
    return dict(pos=pos, vel=vel, mass=mass, ndm=None, nstar=None)
