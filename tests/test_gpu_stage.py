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


@pytest.mark.parametrize("cplx", [False, True])
def test_large_non_finite_amplitudes_are_refused(cplx):
    """Amplitudes beyond the staged size come back bit by bit, and a non-finite T2, found on
    the device, is refused with the current amplitudes unchanged."""
    import numpy as np
    from cc4s_b200 import CoupledClusterError, Solver
    from oracle import inputs
    o, v = 16, 91   # (o v)^2 = 2119936 > 2^21
    s = inputs.synthetic_system(o, v, 8, complex=cplx, seed=1)
    rng = np.random.default_rng(2)
    T = [rng.standard_normal(n) for n in ((v, o), (v, v, o, o))]
    if cplx:
        T = [t + 1j * rng.standard_normal(t.shape) for t in T]
    sol = Solver({})
    sol.set_inputs(s.eps_h, s.eps_p, s.gamma, half_grid=not cplx)
    for _ in range(9):  # enough transfers for the pinned buffers
        sol.set_initial_amplitudes(*T)
        for x, y in zip(sol.amplitudes(), T):
            np.testing.assert_array_equal(x, y)
    for at in ((0, 0, 0, 0), (v - 1, v - 1, o - 1, o - 1)):
        bad = T[1].copy()
        bad[at] = complex(0.0, np.inf) if cplx else np.nan
        with pytest.raises(CoupledClusterError) as e:
            sol.set_initial_amplitudes(T[0], bad)
        assert e.value.status == 9
        for x, y in zip(sol.amplitudes(), T):
            np.testing.assert_array_equal(x, y)
    sol.close()
