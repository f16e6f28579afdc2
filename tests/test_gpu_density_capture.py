"""The fixed-list density and its adjoint on one thread while another thread
captures a CUDA graph: neither disturbs the other, in a fresh process (the first
call sets up the packed rows' memory) and in later calls."""
import os
import subprocess
import sys

import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

CHILD = r"""
import sys, threading
import ctypes as C
import torch
from ahop_b200 import autograd
n = 40000
pos = torch.rand(n, 3, dtype=torch.float64, device="cuda") - 0.5
mass = torch.ones(n, dtype=torch.float64, device="cuda")
nei = torch.randint(0, n, (n, 8), dtype=torch.int32, device="cuda")
nei[:, 7] = (torch.arange(n, device="cuda") + 1) % n
dens = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]
grad = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
lib = autograd._bind()
prm = autograd.AhopAdjParams(8, 0, 1.0, 1.0, 1.0)
side = torch.cuda.Stream()
x = torch.zeros(1, device="cuda")
x += 1
torch.cuda.synchronize()
codes = []

def call(out):
    st = C.c_void_p(side.cuda_stream)
    codes.append(lib.ahop_density_fixed(C.byref(prm), pos.data_ptr(), mass.data_ptr(), nei.data_ptr(), n,
                                        out.data_ptr(), st))
    codes.append(lib.ahop_density_adjoint(C.byref(prm), pos.data_ptr(), mass.data_ptr(), nei.data_ptr(), n,
                                          out.data_ptr(), grad.data_ptr(), st))

for k in range(2):
    g = torch.cuda.CUDAGraph()
    try:
        with torch.cuda.graph(g):
            x += 1
            t = threading.Thread(target=call, args=(dens[k],))
            t.start()
            t.join()
            x += 1
    except Exception as e:
        sys.exit(f"capture {k} ended: {codes} {lib.ahop_last_error()} {e}")
    g.replay()
torch.cuda.synchronize()
call(dens[2])
torch.cuda.synchronize()
assert codes == [0] * 6, (codes, lib.ahop_last_error())
assert float(x) == 5.0
assert torch.equal(dens[0], dens[2]) and torch.equal(dens[1], dens[2])
assert bool((dens[2] > 0).all())
"""


def test_beside_a_capture():
    if not gpu_available():
        pytest.skip("no CUDA device")
    from ahop_b200 import build
    lib = build.build()
    env = dict(os.environ, PYTHONPATH=os.path.dirname(os.path.dirname(lib)))
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=240)
    assert r.returncode == 0, r.stderr[-2000:]
