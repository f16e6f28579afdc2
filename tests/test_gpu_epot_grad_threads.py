"""Potential gradients from two threads on two streams: one whose stream is busy
does not hold up the other, and both get what a call alone gets."""
import ctypes as C
import threading
import time

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


def test_two_streams():
    import torch
    from ahop_b200 import _lib, autograd, halo_props
    lib = autograd._bind()
    rng = np.random.default_rng(4)
    sizes = np.array([900, 2000, 40, 1])
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(off[-1])
    dev = torch.device("cuda:0")
    d_off = torch.from_numpy(off).to(dev)
    mass = torch.ones(n, dtype=torch.float64, device=dev)
    centre = torch.zeros(4, dtype=torch.int32, device=dev)
    gh = torch.ones(4, dtype=torch.float64, device=dev)
    pos = [torch.from_numpy(0.01 * rng.normal(size=(n, 3))).to(dev) for _ in range(2)]
    prm = halo_props.params(1.0, 0.0, 1.0, True, 1)
    streams = [torch.cuda.Stream() for _ in range(2)]
    took = [0.0, 0.0]

    def call(k, out, st):
        t = time.perf_counter()
        _lib.check(lib.ahop_epot_grad(C.byref(prm), d_off.data_ptr(), off.ctypes.data, 4, pos[k].data_ptr(),
                                      mass.data_ptr(), centre.data_ptr(), gh.data_ptr(), out.data_ptr(),
                                      C.c_void_p(st.cuda_stream)), "epot_grad")
        took[k] = time.perf_counter() - t

    want = []
    for k in range(2):
        g = torch.zeros_like(pos[k])
        torch.cuda.synchronize()
        call(k, g, streams[k])
        want.append(g)

    for rep in range(2):  # the first round may allocate
        got = [torch.zeros_like(p) for p in pos]
        torch.cuda.synchronize()
        with torch.cuda.stream(streams[0]):
            torch.cuda._sleep(int(1.5e9))  # most of a second
        th = threading.Thread(target=call, args=(0, got[0], streams[0]))
        th.start()
        time.sleep(0.05)
        call(1, got[1], streams[1])
        th.join()
        torch.cuda.synchronize()
        for k in range(2):
            assert torch.equal(got[k], want[k])
    assert took[1] < 0.25 * took[0], took
