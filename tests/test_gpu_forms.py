"""The digit-form contractions on general operands on a B200 (tests/kernels/forms_check.cu):
two-level views in every order of the strides, second outputs, planar complex products, sliced
operands with runs of rows, and blocks that eight digits leave to the FP64 pipe."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(os.path.dirname(__file__), "kernels"))


def test_forms():
    import build as kbuild
    r = subprocess.run([kbuild.build("forms_check")], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert " 0 failures" in r.stdout
