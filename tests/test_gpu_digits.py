"""The digit-form contraction kernels (four digits: split precision, eight: FP64) at the
edges of their tiles (128 x 128 and 128 x 64), of the K step of 32 and of the K blocks of
64, over several ranges of k and beyond one S32 accumulation span (16384 of K in one range),
on rows graded along k and with a non-finite input, against 128-bit dot products with a derived bound, relative to
sum |a b| where the form stands for FP64 (tests/kernels/digits_check.cu)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(os.path.dirname(__file__), "kernels"))


@pytest.mark.parametrize("shape", [
    (1, 1, 1, 0, 0), (128, 64, 32, 0, 1), (129, 65, 33, 1, 0), (127, 191, 97, 0, 0),
    (300, 520, 160, 1, 1), (2500, 1300, 64, 0, 0), (130, 70, 16417, 1, 0), (2100, 2100, 16417, 0, 0)])
def test_digit_forms(shape):
    import build as kbuild
    exe = kbuild.build("digits_check")
    r = subprocess.run([exe] + [str(x) for x in shape], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.count("errflag=0") == 12
    # an output of few tiles shares the SMs out over k; one of many drains a tile twice
    several, spans = shape[2] > 16384 and shape[0] < 1000, 2 if shape[0] == 2100 else 1
    assert r.stdout.count("parts=1 ") == (0 if several else 2)
    assert r.stdout.count("spans=%d\n" % spans) == 2
