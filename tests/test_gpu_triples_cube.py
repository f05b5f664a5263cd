"""The (T) energy where its hole cubes still fit shared memory (o up to 29) and one beyond,
and at the smallest sizes, with ragged last blocks, against the oracle (the tolerance of
test_gpu_triples.py: the sums differ in order only)."""
import warnings

import numpy as np
import pytest

from oracle import inputs, triples

pytestmark = pytest.mark.gpu
warnings.simplefilter("ignore")


@pytest.mark.parametrize("shape,block", [((1, 5, 8), 2), ((2, 3, 7), 0), ((17, 5, 40), 2),
                                         ((29, 4, 30), 3), ((30, 4, 30), 3)])
def test_triples_cubes(shape, block):
    from cc4s_b200 import Solver
    No, Nv, NG = shape
    s = inputs.synthetic_system(No, Nv, NG, seed=No * Nv)
    rng = np.random.default_rng(NG)
    T1 = rng.standard_normal((Nv, No)) * 0.03
    T2 = rng.standard_normal((Nv, Nv, No, No)) * 0.03
    T2 = T2 + T2.transpose(1, 0, 3, 2)
    ref = triples.triples_reference(T1, T2, triples.triples_integrals(s), s.eps_h, s.eps_p)
    sol = Solver({})
    try:
        sol.set_inputs(s.eps_h, s.eps_p, s.gamma, half_grid=True)
        sol.set_initial_amplitudes(T1, T2)
        r = sol.perturbative_triples(block)
    finally:
        sol.close()
    # With one hole the energy vanishes, (4/3 - 2 + 2/3) W S / D = 0, and both sides are
    # rounding: a few 2^-53 of sum |W S / D|, below 1e-3 at these amplitudes (0.03 each).
    assert abs(r["correlation"] - ref) < 1e-11 * abs(ref) + 4 * 2.0 ** -53 * 1e-3, \
        (r["correlation"], ref)
