"""ahop_release_device_memory between opening part files and decoding them: the
open reader keeps what it has staged."""
import ctypes as C
import os
import sys

import numpy as np
import pytest

from conftest import gpu_available

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
import ramses_files  # noqa: E402
import ramses_oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not gpu_available():
        pytest.skip("no CUDA device")
    from ahop_b200 import build
    build.build()


def test_release_between_open_and_decode(tmp_path):
    import torch
    from ahop_b200 import _lib, ramses
    n = 40000
    P = ramses_files.make_particles(61, 4, n - 3000, 2000, 1000)
    paths = ramses_files.write_arrays(str(tmp_path), P, 4, [0, 15000, n])
    want = ramses_oracle.read_parts(paths, 4, "all", 2.0, 3.0)
    ramses.read_parts(paths, 4, "all", 2.0, 3.0)  # binds the entry points; leaves the staging kept
    lib = _lib.lib()
    arr = (C.c_char_p * len(paths))(*[os.fsencode(p) for p in paths])
    prm = ramses.AhopRamsesParams(4, 0, 2.0, 3.0)
    cnt = ramses.AhopRamsesCounts()
    _lib.check(lib.ahop_ramses_open(arr, len(paths), C.byref(prm), C.byref(cnt)), "open")
    try:
        _lib.check(lib.ahop_release_device_memory(), "release")
        k = int(cnt.nselected)
        assert k == want["nselected"]
        out = {f: torch.empty((k, 3) if f != "mass" else k, dtype=torch.float64, device="cuda")
               for f in ("pos", "vel", "mass")}
        _lib.check(lib.ahop_ramses_decode_device(out["pos"].data_ptr(), out["vel"].data_ptr(), out["mass"].data_ptr(),
                                                 None, torch.cuda.current_stream().cuda_stream), "decode")
        torch.cuda.synchronize()
    finally:
        lib.ahop_ramses_close()
    for f in out:
        assert np.array_equal(out[f].cpu().numpy(), want[f]), f
    # closed: everything goes back (the pinned pieces aside, device memory is what is counted)
    _lib.check(lib.ahop_release_device_memory(), "release")
    ramses.read_parts(paths, 4, "all", 2.0, 3.0)
