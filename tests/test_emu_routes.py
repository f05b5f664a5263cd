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
    lib.emu_split_count.restype = lib.emu_alloc_failures.restype = ctypes.c_uint64
    lib.emu_live_bytes.restype = lib.emu_peak_bytes.restype = ctypes.c_size_t
    lib.emu_force_digits(1)
    yield lib
    lib.emu_force_digits(0)
    lib.emu_fail_split_in(-1)


def _limit(lib, single=0, total=0):
    lib.emu_alloc_limit(ctypes.c_size_t(single), ctypes.c_size_t(total))


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


def _product(emu, A, B, digits):
    M, K = A.shape
    C = np.zeros((M, B.shape[1]))
    P = ctypes.POINTER(ctypes.c_double)
    A, B = np.ascontiguousarray(A), np.ascontiguousarray(B)
    emu.emu_gemm_split(A.ctypes.data_as(P), B.ctypes.data_as(P), C.ctypes.data_as(P),
                       ctypes.c_int64(M), ctypes.c_int64(C.shape[1]), ctypes.c_int64(K), digits)
    return C


def _graded(kind, rng, M, N, K):
    """Operands that the eight-digit form (62 bits below the largest element of a row) must
    not lose against FP64, and some on which it holds anyway."""
    A, B = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    name, _, x = kind.partition(" ")
    x = float(x or 0)
    if name == "opposed":    # A falls along k, B rises
        w = x ** (-np.arange(K) / (K - 1))
        A, B = A * w, B * w[::-1, None]
    elif name == "alike":    # both fall
        w = x ** (-np.arange(K) / (K - 1))
        A, B = A * w, B * w[:, None]
    elif name == "rows":     # eight rows of A against a rising B, the others even
        w = x ** (-np.arange(K) / (K - 1))
        A[16:24] *= w
        B = B * w[::-1, None]
    elif name == "blocks":   # the large elements of either meet tiny ones of the other
        q = K // 4
        A *= x
        B *= x
        A[:, :q], B[:q] = rng.uniform(.5, 1, (M, q)), 1e-13
        A[:, -q:], B[-q:] = 1e-13, rng.uniform(.5, 1, (q, N))
    elif name == "spike":    # one element per column far above the others
        B[rng.integers(K, size=N), np.arange(N)] = x
    elif name == "scaled":   # rows of very different magnitude, which a row scale absorbs
        A *= x ** rng.uniform(-1, 1, (M, 1))
    elif name == "extreme":  # beyond the exponents that the scaling is used for
        A[5] *= x
    elif name == "zeros":
        A[3], B[:, 7] = 0.0, 0.0
        A[rng.random(A.shape) < 0.5] = 0.0
    return A, B


@pytest.mark.parametrize("kind,refuses", [
    ("even", False), ("opposed 30", False), ("opposed 1e3", True), ("opposed 1e6", True),
    ("opposed 1e12", True), ("alike 1e8", False), ("rows 1e8", True), ("blocks 1e-3", True),
    ("spike 100", False), ("scaled 1e30", False), ("extreme 1e-150", True), ("zeros", False)])
@pytest.mark.parametrize("shape", [(64, 64, 64), (96, 130, 256)])
def test_eight_digits_are_no_less_precise_than_fp64(emu, kind, refuses, shape):
    """Against 80-bit sums: the error relative to sum |a b| of each output and the 2-norm of
    all errors stay within what the plain FP64 chain shows on the same operands (1.25 times
    its largest, and not below one rounding of the result)."""
    rng = np.random.default_rng(11)
    A, B = _graded(kind, rng, *shape)
    Al = A.astype(np.longdouble)
    ref, total = Al @ B.astype(np.longdouble), np.abs(Al) @ np.abs(B)
    before = emu.emu_refused_count()
    eight, chain = _product(emu, A, B, 8), _product(emu, A, B, 0)
    assert (emu.emu_refused_count() > before) == refuses

    def worst(C):
        return float((np.abs(C - ref) / np.where(total > 0, total, 1)).max())

    def norm(C):
        return float(np.linalg.norm(((C - ref) / np.where(total > 0, total, 1)).astype(float)))
    u = 2.0 ** -53
    assert worst(eight) <= max(1.25 * worst(chain), u)
    assert norm(eight) <= max(1.1 * norm(chain), u)


def test_eight_digits_keep_non_finite_elements_to_their_outputs(emu):
    """An Inf or NaN shows where the FP64 chain shows it, and nowhere else."""
    rng = np.random.default_rng(2)
    A, B = rng.standard_normal((70, 64)), rng.standard_normal((64, 66))
    A[3, 5], A[40, 7], B[9, 2] = np.inf, np.nan, -np.inf
    B[5, 60] = 0.0
    eight, chain = _product(emu, A, B, 8), _product(emu, A, B, 0)
    np.testing.assert_array_equal(np.isnan(eight), np.isnan(chain))
    np.testing.assert_array_equal(np.isinf(eight), np.isinf(chain))


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("slice_size", [0, 8])
def test_residual_in_eight_digits_matches_oracle(emu, cplx, slice_size):
    """Every eligible contraction of the FP64 residual in the digit form (ladder with its
    shared X panel, planar complex contractions of both kinds): within rounding of the
    oracle's, and different from the FP64 pipe's (the digit form really ran)."""
    from oracle import ccsd
    rng = np.random.default_rng(5)
    n = NO + NV
    if cplx:
        g = rng.standard_normal((NG, n, n)) + 1j * rng.standard_normal((NG, n, n))
        g = 0.1 * (g + g.conj().transpose(0, 2, 1))
    else:
        g = rng.standard_normal((NG, n, n)) * 0.1
        g = g + g.transpose(0, 2, 1)
    s = inputs.System(np.sort(rng.uniform(-1.5, -.5, NO)), np.sort(rng.uniform(.2, 3, NV)), g,
                      half_grid=not cplx)
    T = _amplitudes(cplx)
    out = []
    for forced in (1, 0):
        from cc4s_b200 import Solver
        emu.emu_force_digits(forced)
        sol = Solver({"integralsSliceSize": slice_size} if slice_size else {}, lib=emu._name)
        sol.set_inputs(s.eps_h, s.eps_p, s.gamma, half_grid=not cplx)
        out.append(sol.residual(T))
        sol.close()
    kw = dict(slice_size=slice_size) if slice_size and cplx else {}
    Q = ccsd.residuum(T, ccsd.CcsdInputs(s), **kw)
    for q in range(2):
        assert np.abs(out[0][q] - Q[q]).max() < 1e-13 * np.abs(Q[q]).max()
    assert np.abs(out[0][1] - out[1][1]).max() > 0.0


@pytest.mark.parametrize("cplx", [False, True])
def test_fp64_runs_without_room_for_the_digits(emu, cplx):
    """FP64 needs no digit scratch: where the device has no room for some of it (the ladder's
    shared X panel with its per-contraction part, the larger contractions), the residual is
    the oracle's all the same, what fits still runs in digits, and a size that did not fit is
    not tried for again by every contraction of the call."""
    from oracle import ccsd
    o, v, G = 8, 24, 64
    s = inputs.synthetic_system(o, v, G, complex=cplx, seed=3)
    rng = np.random.default_rng(5)
    T1 = rng.standard_normal((v, o)) * 0.02
    T2 = rng.standard_normal((v, v, o, o)) * 0.02
    T2 = T2 + T2.transpose(1, 0, 3, 2)
    from cc4s_b200 import Solver
    # the ladder's block size only trades memory for speed on the real path
    sol = Solver({} if cplx else {"integralsSliceSize": 8}, lib=emu._name)
    sol.set_inputs(s.eps_h, s.eps_p, s.gamma, half_grid=not cplx)
    # above the amplitude vectors (n1^2 = 36864 values per plane), below the largest scratch
    _limit(emu, 40000 * 8 * (2 if cplx else 1))
    try:
        for _ in range(2):
            f0, c0 = emu.emu_alloc_failures(), emu.emu_split_count()
            R = sol.residual((T1, T2))
            assert 1 <= emu.emu_alloc_failures() - f0 <= 4
            assert emu.emu_split_count() > c0
    finally:
        _limit(emu)
        sol.close()
    Q = ccsd.residuum((T1, T2), ccsd.CcsdInputs(s))
    for q in range(2):
        assert np.abs(R[q] - Q[q]).max() < 1e-13 * np.abs(Q[q]).max()


@pytest.mark.parametrize("kind", ["real", "stacked", "complex"])
def test_vertex_adjoint_without_room_for_a_device_copy(emu, kind):
    """The vertex adjoint is put together on the host, with the same values, where the device
    has no room for a copy of the whole vertex."""
    emu.emu_force_digits(0)
    from cc4s_b200 import Solver
    s = _system(cplx=kind != "real")
    sol = Solver({}, lib=emu._name)
    sol.set_inputs(s.eps_h, s.eps_p, s.gamma, half_grid=kind != "complex")
    args = (_amplitudes(kind == "complex"), _amplitudes(kind == "complex", seed=4))
    _, ref = sol.residual_vjp(*args)
    f0 = emu.emu_alloc_failures()
    planes = 1 if kind == "real" else 2   # above every block, below the whole vertex
    _limit(emu, 8 * planes * NG * (NV * NV + (NO + NV) ** 2) // 2)
    try:
        _, g = sol.residual_vjp(*args)
    finally:
        _limit(emu)
        sol.close()
    assert emu.emu_alloc_failures() == f0 + 1
    np.testing.assert_array_equal(g, ref)


def test_complex_ladder_slab_stays_within_the_caller_and_the_device(emu):
    """The complex ladder contracts several slices together where it may: not where
    integralsSliceSize bounds the slab, and not where the device has no room; the residual is
    the same."""
    emu.emu_force_digits(0)
    from cc4s_b200 import Solver
    s = _system(cplx=True)
    T = _amplitudes(cplx=True)

    def residual(limit=0, **options):
        sol = Solver(options, lib=emu._name)
        base = emu.emu_live_bytes()
        emu.emu_peak_bytes(1)
        _limit(emu, total=limit and base + limit)
        try:
            sol.set_inputs(s.eps_h, s.eps_p, s.gamma, half_grid=False)
            peak, live = emu.emu_peak_bytes(0) - base, emu.emu_live_bytes() - base
        finally:
            _limit(emu)
        R = sol.residual(T)
        if not limit and not options:   # the adjoint schedule too
            sol.residual_vjp(T, T, gradient=False)
        sol.close()
        return R, peak, live
    ref, peak1, live1 = residual()
    one, peak0, live0 = residual(integralsSliceSize=NO)   # the default slices, one by one
    slice_bytes = 16 * NO * NO * NV * NV
    groups = NV // NO - 1
    assert live1 - live0 == (groups - 1) * slice_bytes
    tight, peak, live = residual(limit=max(peak0, live0) + 1024)
    assert live == live0
    for q in range(2):
        assert np.abs(one[q] - ref[q]).max() < 1e-13 * np.abs(ref[q]).max()
        np.testing.assert_array_equal(tight[q], one[q])


def test_profile_tells_the_forms_apart(emu, monkeypatch, tmp_path):
    """An FP64 profile counts no split-precision launches, the slicing of the ladder's shared
    panel included, and the log names the digit form."""
    from cc4s_b200 import Solver
    s = inputs.synthetic_system(8, 24, 64, seed=3)
    rng = np.random.default_rng(5)
    T2 = rng.standard_normal((24, 24, 8, 8)) * 0.02
    T = rng.standard_normal((24, 8)) * 0.02, T2 + T2.transpose(1, 0, 3, 2)
    for precision, kind in (("fp64", "digits8"), ("split3", "split")):
        log = tmp_path / precision
        monkeypatch.setenv("CC4S_PROFILE_LOG", str(log))
        sol = Solver({"precision": precision, "integralsSliceSize": 8, "profile": True},
                     lib=emu._name)
        sol.set_inputs(s.eps_h, s.eps_p, s.gamma)
        sol.residual(T)
        n = sol.stats()["split_launches"]
        sol.close()
        kinds = {line.split()[0] for line in log.read_text().splitlines() if line[0] != "#"}
        assert kind in kinds and "dmma" in kinds
        assert (n > 0) == (precision == "split3")
        assert precision == "split3" or "split" not in kinds


@pytest.mark.parametrize("cplx,shape,block", [(False, (12, 5, 9), 4), (True, (10, 5, 9), 4),
                                              (False, (2, 63, 20), 16), (True, (2, 63, 20), 16)])
def test_triples_cubes_and_operands_sliced_in_eight_digits(emu, cplx, shape, block):
    """(T) where the energy adds the singles (hole cubes), and where FP64 operands are sliced
    once, against the oracle; operands that eight digits refuse run on the FP64 pipe, with
    the same agreement."""
    from cc4s_b200 import Solver
    from oracle import triples
    No, Nv, NGs = shape
    s = inputs.synthetic_system(No, Nv, NGs, complex=cplx, seed=6)
    rng = np.random.default_rng(3)
    T1 = rng.standard_normal((Nv, No)) * 0.03
    T2 = rng.standard_normal((Nv, Nv, No, No)) * 0.02
    if cplx:
        T1 = T1 + 1j * rng.standard_normal(T1.shape) * 0.03
        T2 = T2 + 1j * rng.standard_normal(T2.shape) * 0.02
    T2 = T2 + T2.transpose(1, 0, 3, 2)
    for graded in (False, True):
        if graded:  # T falls along the virtual index that the contractions sum over
            w = 1e-9 ** (np.arange(Nv) / (Nv - 1))
            T2 = T2 * w[:, None, None, None] * w[None, :, None, None]
        ref = triples.triples_reference(T1, T2, triples.triples_integrals(s), s.eps_h, s.eps_p)
        sol = Solver({}, lib=emu._name)
        sol.set_inputs(s.eps_h, s.eps_p, s.gamma, half_grid=not cplx)
        sol.set_initial_amplitudes(T1, T2)
        before = emu.emu_split_count()
        e = sol.perturbative_triples(block, reference_form=True)["correlation"]
        used = emu.emu_split_count() - before
        sol.close()
        assert abs(e - ref) < 1e-11 * abs(ref), (e, ref)
        assert Nv < 60 or (used > 0) == (not graded)
