"""The (T) energy at the smallest number of holes that takes the hole cubes (12, complex 10),
where they still fit shared memory (29, complex 23) and one beyond, below and at the smallest
block (4 orbitals), with ragged last blocks, and with operands sliced once in eight digits,
against the oracle (the tolerance of test_gpu_triples.py: the sums differ in order only)."""
import warnings

import numpy as np
import pytest

from oracle import inputs, triples

pytestmark = pytest.mark.gpu
warnings.simplefilter("ignore")


@pytest.mark.parametrize("shape,block", [((1, 5, 8), 2), ((2, 3, 7), 0), ((17, 5, 40), 2),
                                         ((29, 4, 30), 3), ((30, 4, 30), 3), ((12, 6, 20), 4),
                                         ((17, 5, 40), 4), ((29, 4, 30), 0), ((30, 4, 30), 0),
                                         ((4, 61, 50), 8), ((3, 62, 40), 0)])
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


@pytest.mark.parametrize("shape,block", [((10, 6, 20), 4), ((13, 5, 16), 0), ((23, 4, 12), 4),
                                         ((24, 4, 12), 4), ((9, 6, 20), 4), ((3, 62, 30), 11)])
def test_triples_cubes_complex(shape, block):
    from cc4s_b200 import Solver
    No, Nv, NG = shape
    s = inputs.synthetic_system(No, Nv, NG, complex=True, seed=No * Nv)
    rng = np.random.default_rng(NG)

    def amplitudes(*n):
        return (rng.standard_normal(n) + 1j * rng.standard_normal(n)) * 0.02
    T1, T2 = amplitudes(Nv, No), amplitudes(Nv, Nv, No, No)
    T2 = T2 + T2.transpose(1, 0, 3, 2)
    V = triples.triples_integrals(s)
    sol = Solver({})
    try:
        sol.set_inputs(s.eps_h, s.eps_p, s.gamma, half_grid=False)
        sol.set_initial_amplitudes(T1, T2)
        for form in (False, True):
            f = triples.triples_reference if form else triples.triples_atrip
            if not form and (No > 13 or Nv > 20):
                continue  # the tuple loop of the oracle takes minutes
            ref = f(T1, T2, V, s.eps_h, s.eps_p)
            e = sol.perturbative_triples(block, reference_form=form)["correlation"]
            assert abs(e - ref) < 1e-11 * abs(ref), (e, ref)
    finally:
        sol.close()
