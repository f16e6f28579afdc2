"""The part-file reader on files whose payloads fill one piece of the staging
buffers exactly, hold one particle, none, and need several pieces, read twice
(the second call reuses the buffers), against the CPU restatement; and a file
that ends inside a payload."""
import os
import sys

import numpy as np
import pytest

from conftest import gpu_available

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
import ramses_files  # noqa: E402
import ramses_oracle  # noqa: E402

pytestmark = pytest.mark.gpu

PIECE = 524288  # doubles of one piece


@pytest.fixture(scope="module", autouse=True)
def _built():
    if not gpu_available():
        pytest.skip("no CUDA device")
    from ahop_b200 import build
    build.build()


@pytest.mark.parametrize("version", [3, 4])
def test_pieces(tmp_path, version):
    from ahop_b200 import ramses
    n = 3 * PIECE + 12345
    P = ramses_files.make_particles(51, version, n - 70000, 60000, 10000)
    paths = ramses_files.write_arrays(str(tmp_path), P, version, [0, PIECE, PIECE, PIECE + 1, n])
    want = ramses_oracle.read_parts(paths, version, "all", 2.0, 3.0)
    for k in range(3):
        if k == 1:  # another set in between leaves other bytes in the buffers
            Q = ramses_files.make_particles(53, version, 40000, 0, 0)
            ramses.read_parts(ramses_files.write_arrays(str(tmp_path / "q"), Q, version, [0, 40000]), version, "all")
            continue
        got = ramses.read_parts(paths, version, "all", 2.0, 3.0)
        assert got["nselected"] == want["nselected"]
        for f in ("pos", "vel", "mass"):
            assert np.array_equal(got[f].cpu().numpy(), want[f]), f


def test_truncated_payload(tmp_path):
    from ahop_b200 import ramses
    from ahop_b200._lib import AhopError
    P = ramses_files.make_particles(52, 4, 5000, 500, 0)
    paths = ramses_files.write_arrays(str(tmp_path), P, 4, [0, 3000, 5500])
    with open(paths[1], "r+b") as f:
        f.truncate(20000)
    with pytest.raises(AhopError, match="EDATA"):
        ramses.read_parts(paths, 4, "all", 2.0, 3.0)
