"""The digit-form routes of the product's schedules on the CPU emulation of the device
operations (tests/emu/ops_emu.cpp), whose test controls force them at small sizes."""
import ctypes
import os
import sys

import numpy as np
import pytest

from oracle import inputs

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "emu"))

NO, NV, NG = 4, 16, 64
TIMEOUT = 7


@pytest.fixture()
def emu():
    import build_emu
    from cc4s_b200 import _abi
    lib = _abi.load(build_emu.build())
    lib.emu_split_count.restype = ctypes.c_uint64
    lib.emu_force_digits(1)
    yield lib
    lib.emu_force_digits(0)
    lib.emu_fail_split_in(-1)


def _system(cplx=False, seed=7):
    return inputs.synthetic_system(NO, NV, NG, complex=cplx, seed=seed)


def _amplitudes(cplx=False, seed=3):
    rng = np.random.default_rng(seed)
    T1 = rng.standard_normal((NV, NO)) * 0.01
    T2 = rng.standard_normal((NV, NV, NO, NO)) * 0.01
    if cplx:
        T1 = T1 + 1j * rng.standard_normal(T1.shape) * 0.01
        T2 = T2 + 1j * rng.standard_normal(T2.shape) * 0.01
    return T1, T2 + T2.transpose(1, 0, 3, 2)


def _solver(lib, precision="fp64", cplx=False, **options):
    from cc4s_b200 import Solver
    s = _system(cplx)
    sol = Solver(dict(precision=precision, maxIterations=2, energyConvergence=1e-300,
                      amplitudesConvergence=1e-300, **options), lib=lib._name)
    sol.set_inputs(s.eps_h, s.eps_p, s.gamma, half_grid=not cplx)
    return sol


def _lattice(n=5):
    B = 2 * np.pi / 5.0 * np.eye(3)
    r = np.arange(n) - n // 2
    return B, np.array([(a, b, c) for c in r for b in r for a in r], dtype=float) @ B


def _fsc(sol):
    B, grid = _lattice()
    U = np.random.default_rng(1).standard_normal((len(grid), NG)) + 0j
    return sol.finite_size_correction(grid, B, U, np.ones(len(grid)), grid_size=2)


ENTRIES = {
    "run": lambda sol: sol.run(),
    "residual": lambda sol: sol.residual(_amplitudes()),
    "backward": lambda sol: sol.backward(),
    "vjp": lambda sol: sol.residual_vjp(_amplitudes(), _amplitudes(seed=4)),
    "relaxed": lambda sol: sol.relaxed_gradient(max_iterations=2),
    "triples": lambda sol: sol.perturbative_triples(),
    "fsc": _fsc,
}


@pytest.mark.parametrize("precision", ["fp64", "split3"])
@pytest.mark.parametrize("entry", sorted(ENTRIES))
def test_expired_wait_reaches_the_caller(emu, entry, precision):
    """A tensor-core kernel that gives up a bounded wait leaves its output incomplete: the
    entry point that ran it reports a timeout, whichever contraction it was, and the handle
    stays unusable until its inputs are set again."""
    from cc4s_b200 import CoupledClusterError
    sol = _solver(emu, precision)
    sol.set_initial_amplitudes(*_amplitudes())
    before = emu.emu_split_count()
    ENTRIES[entry](sol)
    count = emu.emu_split_count() - before
    sol.close()
    assert count > 0
    for at in {0, count // 2, count - 1}:
        sol = _solver(emu, precision)
        sol.set_initial_amplitudes(*_amplitudes())
        emu.emu_fail_split_in(at)
        with pytest.raises(CoupledClusterError) as e:
            ENTRIES[entry](sol)
        assert e.value.status == TIMEOUT, at
        sol.close()


def test_expired_wait_outlives_the_growing_of_the_scratch(emu):
    """The record is kept when a later contraction of the same call needs more scratch, and
    for later calls."""
    from cc4s_b200 import CoupledClusterError
    sol = _solver(emu)
    emu.emu_fail_split_in(0)
    for _ in range(2):
        with pytest.raises(CoupledClusterError) as e:
            sol.residual(_amplitudes())
        assert e.value.status == TIMEOUT
    s = _system()
    sol.set_inputs(s.eps_h, s.eps_p, s.gamma)
    sol.residual(_amplitudes())
    sol.close()


def test_expired_wait_while_the_integrals_are_built(emu):
    from cc4s_b200 import CoupledClusterError
    emu.emu_fail_split_in(0)
    with pytest.raises(CoupledClusterError) as e:
        _solver(emu)
    assert e.value.status == TIMEOUT
