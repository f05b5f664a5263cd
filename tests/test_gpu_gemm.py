"""The FP64 tensor-pipe contraction in each of its tile shapes (N up to 16, up to 32, 64 x 64,
128 x 128, narrow M transposed), at their edges and with split K, against 128-bit dot
products within the rounding bound (tests/kernels/gemm_check.cu)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(os.path.dirname(__file__), "kernels"))


@pytest.mark.parametrize("shape", [
    (1, 1, 1, 3, 0, 0), (65, 16, 33, 5, 0, 1), (64, 17, 16, 4, 1, 0), (7, 300, 40, 6, 0, 0),
    (16, 16, 40000, 1, 1, 0), (130, 1, 2049, 1, 0, 0), (32, 33, 65, 2, 1, 1),
    (171, 171, 19, 9, 0, 0), (129, 257, 100, 1, 0, 1), (1500, 1400, 65, 1, 1, 0)])
def test_gemm_tiles(shape):
    import build as kbuild
    exe = kbuild.build("gemm_check")
    r = subprocess.run([exe] + [str(x) for x in shape], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.count("ok") == 4
