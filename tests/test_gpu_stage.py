"""The staged host transfers on a B200: values of both strides around the sizes where pinned
buffers come into play, and when those are made (tests/kernels/stage_check.cu)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(os.path.dirname(__file__), "kernels"))


def test_staged_transfers():
    import build as kbuild
    r = subprocess.run([kbuild.build("stage_check")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "ok" in r.stdout
