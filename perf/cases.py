"""Workloads of the CoupledCluster package, called through its public entry points.

Each case is a dict of plain values: ``kind`` (which step), ``No``/``Nv``/``NG``
(holes, particles, vertex rows), ``precision`` (``fp64`` or ``split3``), ``complex``
(complex vertex instead of the real half-grid one) and what the step needs besides.
Systems are seeded random ones with the distributions of ``cc4s_b200/synthetic.py`` and
the vertex scaled by 0.2, on which CCSD converges.

  listed() / draw(rng)      the cases, and more of the same ranges
  prepare(case, seed)       what a program holds before the call
  run(state)                one call
  work, tolerance, exact    its floor, the allowed error, and the result in 64 bits
"""
import math

import numpy as np
import torch

from cc4s_b200 import CoupledCluster, Solver, reference_flops

DEV = "cuda"
F64, C128 = torch.float64, torch.complex128


def listed():
    return [
        # the whole step as the input file names it, on the smallest shipped system:
        # device set-up, upload, iterations and download, bound by latency
        dict(name="step-8-40", kind="step", No=8, Nv=40, NG=200, precision="fp64", complex=False,
             iterations=16),
        # one residual of a molecule in a small basis, odd sizes: the smallest call
        dict(name="residual-5-23", kind="residual", No=5, Nv=23, NG=97, precision="fp64",
             complex=False),
        # CCSD restarted from MP2 amplitudes: an ordinary molecule
        dict(name="ccsd-16-128", kind="ccsd", No=16, Nv=128, NG=512, precision="fp64",
             complex=False, iterations=8),
        # the same in the split form with ragged sizes
        dict(name="ccsd-split-19-171", kind="ccsd", No=19, Nv=171, NG=613, precision="split3",
             complex=False, iterations=8),
        # the package's parity system, and the largest call in each precision
        dict(name="ccsd-32-256", kind="ccsd", No=32, Nv=256, NG=1024, precision="fp64",
             complex=False, iterations=2),
        dict(name="ccsd-split-32-256", kind="ccsd", No=32, Nv=256, NG=1024, precision="split3",
             complex=False, iterations=6),
        # a k-point (complex) vertex in both precisions
        dict(name="ccsd-complex-11-97", kind="ccsd", No=11, Nv=97, NG=310, precision="fp64",
             complex=True, iterations=6),
        dict(name="ccsd-complex-split-16-160", kind="ccsd", No=16, Nv=160, NG=640,
             precision="split3", complex=True, iterations=6),
        # reverse mode: one transposed-Jacobian product with the vertex gradient
        dict(name="vjp-16-128", kind="vjp", No=16, Nv=128, NG=512, precision="fp64",
             complex=False),
        # perturbative triples after CCSD
        dict(name="triples-16-128", kind="triples", No=16, Nv=128, NG=512, precision="fp64",
             complex=False),
        dict(name="triples-split-21-163", kind="triples", No=21, Nv=163, NG=600,
             precision="split3", complex=False),
        # finite-size correction: structure factor and its interpolation
        dict(name="fsc-16-128", kind="fsc", No=16, Nv=128, NG=512, precision="fp64",
             complex=False, shell=13, grid=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Sizes log-uniform between a small molecule and the largest listed system, the
    basis 4 to 10 functions per hole, the vertex 2.5 to 4.5 rows per orbital."""
    kind = rng.choice(["ccsd", "ccsd", "ccsd", "ccsd", "residual", "step", "vjp", "triples",
                       "triples", "fsc"])
    cplx = kind in ("ccsd", "residual", "triples") and rng.random() < 0.3
    precision = rng.choice(["fp64", "split3"]) if kind != "fsc" else "fp64"
    top = {"ccsd": 28, "residual": 20, "step": 16, "vjp": 18, "triples": 20, "fsc": 18}[kind]
    if cplx:
        top = min(top, 13 if kind == "triples" else 16)
    No = _log(rng, 4, top)
    Nv = int(No * rng.uniform(4.0, 10.0 if No < 16 else 8.0))
    Nv = min(Nv, {"triples": 150, "vjp": 160}.get(kind, 230))
    case = dict(kind=kind, No=No, Nv=Nv, NG=int((No + Nv) * rng.uniform(2.5, 4.5)),
                precision=precision, complex=cplx)
    if kind in ("ccsd", "step"):
        case["iterations"] = rng.randint(2, 4 if cplx or No > 20 else 12)
    if kind == "fsc":
        case.update(shell=rng.choice([7, 9, 10, 12]), grid=rng.randint(6, 20))
    return case


# ---- inputs -------------------------------------------------------------------
def _system(case, seed):
    """(eps_h, eps_p, Gamma) as device tensors, Gamma[G, p, q] with p, q the slow axes in
    memory (G fastest), the column-major layout the library takes."""
    o, v, G = case["No"], case["Nv"], case["NG"]
    g = torch.Generator(DEV).manual_seed(seed)
    eh = torch.sort(torch.rand(o, generator=g, device=DEV, dtype=F64) - 1.5).values
    ep = torch.sort(torch.rand(v, generator=g, device=DEV, dtype=F64) * 2.8 + 0.2).values
    n = o + v
    s = 0.2 * 0.1 * G ** -0.25

    def symmetric(sign):
        x = torch.randn(n, n, G, generator=g, device=DEV, dtype=F64)
        upper = torch.triu(torch.ones(n, n, device=DEV, dtype=F64), 0 if sign > 0 else 1)
        x *= upper[:, :, None]
        y = x.transpose(0, 1) * (1 - torch.eye(n, device=DEV, dtype=F64))[:, :, None]
        return x.add_(y, alpha=sign)  # [q][p][G]

    if case["complex"]:
        gam = torch.complex(symmetric(1), symmetric(-1)) * (s / math.sqrt(2.0))
    else:
        gam = symmetric(1) * s
    return eh, ep, gam.permute(2, 1, 0), g


def _pair(G, o):
    """V_abij = sum_G conj(Gamma_ia) Gamma_bj as [a, b, i, j]."""
    A, B = G[:, :o, o:].conj(), G[:, o:, :o]
    v = A.shape[2]
    V = A.permute(2, 1, 0).reshape(v * o, -1) @ B.reshape(B.shape[0], v * o)
    return V.reshape(v, o, v, o).permute(0, 2, 1, 3)


def _denominators(eh, ep):
    d1 = ep[:, None] - eh[None, :]
    return d1, d1[:, None, :, None] + d1[None, :, None, :]


def _amplitudes(case, eh, ep, G, g):
    """A start near the solution: small singles and MP2 doubles."""
    o, v = case["No"], case["Nv"]
    t = torch.randn(v, o, generator=g, device=DEV, dtype=F64) * 0.005
    if case["complex"]:
        t = torch.complex(t, torch.randn(v, o, generator=g, device=DEV, dtype=F64) * 0.005)
    return t, -_pair(G, o) / _denominators(eh, ep)[1]


def _host(x):
    """A numpy array with the first index fastest."""
    order = tuple(reversed(range(x.dim())))
    return x.resolve_conj().permute(order).contiguous().cpu().numpy().transpose(order)


def _lattice(shell):
    """A skewed reciprocal basis and its shell**3 grid vectors around the origin."""
    B = 2 * np.pi / 5.0 * (np.eye(3) + 0.1 * np.array([[0.3, -0.7, 0.4], [0.9, 0.1, -0.5],
                                                       [-0.2, 0.6, -0.8]]))
    r = np.arange(shell) - shell // 2
    idx = np.array([(a, b, c) for c in r for b in r for a in r], dtype=float)
    return B, idx @ B


def _inputs(case, seed):
    """Everything a case's call is given, as device tensors (Gamma in C order for exact)."""
    eh, ep, G, g = _system(case, seed)
    t, T = _amplitudes(case, eh, ep, G, g)
    x = dict(eh=eh, ep=ep, G=G, t=t, T=T)
    if case["kind"] == "vjp":
        x["t_bar"] = torch.randn(t.shape, generator=g, device=DEV, dtype=F64)
        R = torch.randn(T.shape, generator=g, device=DEV, dtype=F64)
        x["T_bar"] = 0.5 * (R + R.permute(1, 0, 3, 2))
    if case["kind"] == "fsc":
        n = case["shell"] ** 3
        U = torch.randn(2, n, case["NG"], generator=g, device=DEV, dtype=F64)
        x["U"] = torch.complex(U[0], U[1]) / math.sqrt(2.0 * case["NG"])
        x["V"] = 0.5 + torch.rand(n, generator=g, device=DEV, dtype=F64)
        x["basis"], x["grid"] = _lattice(case["shell"])
    return x


def _options(case):
    # no convergence test is met, so every pass runs the stated number of iterations
    return dict(precision=case["precision"], maxIterations=case.get("iterations", 16),
                energyConvergence=1e-300, amplitudesConvergence=1e-300)


def prepare(case, seed):
    x = _inputs(case, seed)
    eh, ep, G = x["eh"].cpu().numpy(), x["ep"].cpu().numpy(), _host(x["G"])
    s = dict(kind=case["kind"])
    if case["kind"] == "step":
        s["arguments"] = dict(_options(case), slicedEigenEnergies={"h": eh, "p": ep},
                              coulombVertex=G, halfGrid=True)
    else:
        s["solver"] = Solver(_options(case))
        s["solver"].set_inputs(eh, ep, G, half_grid=not case["complex"])
        s["T"] = (_host(x["t"]), _host(x["T"]))
        if case["kind"] == "vjp":
            s["bar"] = (_host(x["t_bar"]), _host(x["T_bar"]))
        if case["kind"] in ("triples", "fsc"):
            s["solver"].set_initial_amplitudes(*s["T"])
        if case["kind"] == "fsc":
            s.update(U=_host(x["U"]), V=x["V"].cpu().numpy(), grid=x["grid"], basis=x["basis"],
                     n=case["grid"])
    del x
    torch.cuda.empty_cache()  # the library allocates its own device memory
    return s


# ---- one call -----------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "step":
        r = CoupledCluster().run(state["arguments"])
        e, T = r["energy"], r["amplitudes"]
        return dict(energy=np.array([e["correlation"], e["direct"], e["exchange"],
                                     e["secondOrder"]]), T1=T["ph"], T2=T["pphh"])
    s = state["solver"]
    if kind == "ccsd":
        s.set_initial_amplitudes(*state["T"])
        r = s.run()
        T1, T2 = s.amplitudes()
        return dict(energy=np.array([r["correlation"], r["direct"], r["exchange"]]), T1=T1, T2=T2)
    if kind == "residual":
        R1, R2 = s.residual(state["T"])
        return dict(R1=R1, R2=R2)
    if kind == "vjp":
        (t, T), G = s.residual_vjp(state["T"], state["bar"])
        return dict(T1=t, T2=T, vertex=G)
    if kind == "triples":
        r = s.perturbative_triples()
        return dict(energy=np.array([r["correlation"], r["mp2_energy"]]))
    e, S = s.finite_size_correction(state["grid"], state["basis"], state["U"], state["V"],
                                    grid_size=state["n"])
    return dict(energy=np.array([e["uncorrected"], e["corrected"]]), S=S)


# ---- floor and tolerance --------------------------------------------------------
def work(case):
    """The contractions in the formulation with the fewest flops the package counts, and
    every input and output once."""
    o, v, G, kind = case["No"], case["Nv"], case["NG"], case["kind"]
    z = 2 if case["complex"] else 1
    amps, vertex = 8 * z * (o * v + (o * v) ** 2), 8 * z * G * (o + v) ** 2
    iteration = reference_flops(o, v, G, complex=case["complex"])
    if kind in ("ccsd", "step"):
        return dict(bytes=vertex + 2 * amps, flops=case["iterations"] * iteration)
    if kind == "residual":
        return dict(bytes=vertex + 2 * amps, flops=iteration)
    if kind == "vjp":
        return dict(bytes=2 * vertex + 3 * amps, flops=3 * iteration)
    if kind == "triples":
        return dict(bytes=vertex + amps, flops=2.0 * o ** 3 * v ** 3 * (o + v) * z * z)
    n = case["shell"] ** 3
    return dict(bytes=vertex + amps + 16 * n * G,
                flops=2.0 * G * (o * v) ** 2 + 2.0 * G * G * o * v + 8.0 * n * G * G
                + 160.0 * n * (2 * case["grid"]) ** 3)


def tolerance(case):
    """Measured against exact(): FP64 amplitudes within 5e-15 after up to 12 iterations (a
    DIIS system near convergence amplifies rounding further), the split form, which keeps 28
    bits of each operand relative to the largest of its row, within 4e-7."""
    return {"rel": 1e-13} if case["precision"] == "fp64" else {"rel": 2e-6}


# ---- the same in plain 64-bit torch ----------------------------------------------
def _es(spec, *xs):
    return torch.einsum(spec, *xs)


def _residual(t, T, G, o):
    """Spin-restricted CCSD residual over V_pqrs = sum_G conj(Gamma_rp) Gamma_qs."""
    C = G.conj().transpose(1, 2)
    Chh, Cph, Chp, Cpp = C[:, :o, :o], C[:, o:, :o], C[:, :o, o:], C[:, o:, o:]
    Ghh, Gph, Ghp, Gpp = G[:, :o, :o], G[:, o:, :o], G[:, :o, o:], G[:, o:, o:]
    v = t.shape[0]
    X = T + t[:, None, :, None] * t[None, :, None, :]
    V = _es("Gkc,Gld->klcd", Chp, Ghp)
    L = 2 * V - V.transpose(2, 3)
    Kac = -_es("klcd,adkl->ac", L, X)
    Kki = _es("klcd,cdil->ki", L, X)
    j = _es("Gld,dl->G", Ghp, t)
    Lac = Kac + 2 * _es("Gac,G->ac", Cpp, j) - _es("Gak,Gkc->ac", Cpp @ t, Ghp)
    Lki = Kki + 2 * _es("Gki,G->ki", Chh, j) - _es("Gli,Gkl->ki", Chh, Ghp @ t)
    R = _es("ac,cbij->abij", Lac, T) - _es("ki,abkj->abij", Lki, T)
    D = Cph - t @ Chh
    R = R + _es("Gai,Gbj->abij", D, Gpp @ t) - _es("Gai,Gbj->abij", Cph, t @ (Ghh + Ghp @ t))
    D = D + Cpp @ t - 0.5 * _es("Gld,dail->Gai", Chp, X + t[:, None, :, None] * t[None, :, None, :])
    Z = _es("Gai,Gkc->akic", D, Ghp) + _es("lkdc,adil->akic", V - 0.5 * V.transpose(2, 3), T)
    R = R + _es("akic,cbkj->abij", Z, 2 * T - T.transpose(0, 1))
    Dac, Dki = Cpp - t @ Chp, Ghh + Ghp @ t
    Z = _es("Gac,Gki->akci", Dac, Dki) - 0.5 * _es("lkcd,dail->akci", V, T)
    R = R - _es("akci,cbkj->abij", Z, T) - _es("bkci,ackj->abij", Z, T)
    R = R + R.permute(1, 0, 3, 2) + _es("Gai,Gbj->abij", Cph, Gph)
    Z = (_es("Gki,Glj->klij", Chh, Ghh + Ghp @ t) + _es("Glj,Gki->klij", Chh, Ghp @ t))
    R = R + _es("klij,abkl->abij", Z, X) + _es("klij,abkl->abij", _es("klcd,cdij->klij", V, X), T)
    Dbd, flat = Gpp - t @ Ghp, X.reshape(v * v, o * o)
    step = max(1, 400_000_000 // v ** 3)
    parts = []
    for a in range(0, v, step):
        W = _es("Gac,Gbd->abcd", Dac[:, a:a + step], Dbd)
        parts.append((W.reshape(-1, v * v) @ flat).reshape(-1, v, o, o))
    R = R + torch.cat(parts)
    K = _es("klcd,dl->ck", L, t)
    r = Kac @ t - t @ Kki + _es("ck,caki->ai", K, 2 * T - T.transpose(0, 1)) + t @ (K.T @ t)
    r = r + 2 * _es("Gai,G->ai", Cph, j)
    r = r - _es("Gac,Gci->ai", Cpp, _es("ck,Gki->Gci", t, Ghh))
    Y = 2 * X - X.transpose(2, 3)
    r = r + _es("Gac,Gci->ai", Cpp, _es("Gkd,cdik->Gci", Ghp, Y))
    r = r - _es("Gki,Gak->ai", Chh, _es("Glc,ackl->Gak", Ghp, Y))
    return r, R


def _energy(t, T, V):
    X = (T + t[:, None, :, None] * t[None, :, None, :]).conj()
    d, e = 2 * (X * V).sum().real, -(X * V.transpose(2, 3)).sum().real
    return d + e, d, e


def _ccsd(x, case):
    """Jacobi iterations with DIIS of the last four changes (bordered overlap matrix)."""
    o, n, hist = case["No"], case["iterations"], []
    d1, d2 = _denominators(x["eh"], x["ep"])
    V = _pair(x["G"], o)
    first = case["kind"] == "step"
    t, T = (torch.zeros_like(d1), torch.zeros_like(d2)) if first else (x["t"], x["T"])
    second = None
    for it in range(n):
        r, R = (t, V) if first and it == 0 else _residual(t, T, x["G"], o)
        new = torch.cat([(-r / d1).flatten(), (-R / d2).flatten()])
        hist = ([(new, new - torch.cat([t.flatten(), T.flatten()]))] + hist)[:4]
        m = len(hist)
        B = torch.zeros(m + 1, m + 1, device=DEV, dtype=F64)
        B[0, 1:] = B[1:, 0] = -1.0
        for p in range(m):
            for q in range(p, m):
                B[p + 1, q + 1] = B[q + 1, p + 1] = 2 * torch.vdot(hist[p][1], hist[q][1]).real
        rhs = torch.zeros(m + 1, device=DEV, dtype=F64)
        rhs[0] = -1.0
        c = torch.linalg.solve(B, rhs)[1:]
        mix = sum(ck * h[0] for ck, h in zip(c, hist))
        t, T = mix[:d1.numel()].reshape(d1.shape), mix[d1.numel():].reshape(d2.shape)
        if it == 0:
            second = _energy(t, T, V)[0]
    e = list(_energy(t, T, V)) + ([second] if first else [])
    return dict(energy=torch.stack(e), T1=t, T2=T)


def _triples(x, o):
    """(T) energy, one virtual index a at a time: W and the singles of all b, c, i, j, k."""
    t, T, G, eh, ep = x["t"], x["T"], x["G"], x["eh"], x["ep"]
    C = G.conj().transpose(1, 2)
    v = t.shape[0]
    V = _pair(G, o)
    Vh = _es("Gjl,Gkc->jklc", C[:, :o, :o], G[:, :o, o:]).conj().resolve_conj()
    Vp = _es("Gbd,Gck->bcdk", C[:, o:, o:], G[:, o:, :o])
    e = torch.zeros((), device=DEV, dtype=F64)
    de = eh[:, None, None] + eh[None, :, None] + eh[None, None, :]
    for a in range(v):
        A = slice(a, a + 1)
        N = slice(0, v)

        def X(p, q, r, order):  # X_pqr,ijk of one order of the pairs, as [b, c, i, j, k]
            w = _es("pdij,qrdk->pqrijk", T[p], Vp[q][:, r])
            w = w - _es("pqil,jklr->pqrijk", T[p][:, q], Vh[..., r])
            return w.permute(order)[0]

        W = X(A, N, N, (0, 1, 2, 3, 4, 5)) + X(A, N, N, (0, 2, 1, 3, 5, 4))
        W += X(N, A, N, (1, 0, 2, 4, 3, 5)) + X(N, A, N, (1, 2, 0, 4, 5, 3))
        W += X(N, N, A, (2, 0, 1, 5, 3, 4)) + X(N, N, A, (2, 1, 0, 5, 4, 3))
        S = W + _es("i,bcjk->bcijk", t[a], V) + _es("bj,cik->bcijk", t, V[a]) \
            + _es("ck,bij->bcijk", t, V[a])
        D = de[None, None] - ep[a] - (ep[:, None] + ep[None, :])[:, :, None, None, None]
        # S_acbijk = S_abcikj and S_bcaijk = S_abckij by the simultaneous permutations
        Z = 4.0 / 3.0 * S - 2.0 * S.permute(0, 1, 2, 4, 3) + 2.0 / 3.0 * S.permute(0, 1, 3, 4, 2)
        e += ((W.conj() * Z).real / D).sum()
    d2 = _denominators(eh, ep)[1]
    mp2 = -((2 * V - V.transpose(2, 3)) * V.conj() / d2).real.sum()
    return dict(energy=torch.stack([e, mp2]))


def _fsc(x, case):
    """Structure factor with singular vectors, then Catmull-Rom tricubic interpolation of it
    on the lattice box, summed over the refined grid."""
    o, N = case["No"], case["grid"]
    G, X = x["G"].to(C128), x["T"] + x["t"][:, None, :, None] * x["t"][None, :, None, :]
    Y = (2 * X - X.transpose(2, 3)).to(C128)
    W = _es("Fjb,abij->Fai", G[:, :o, o:], Y)
    Q = _es("Fai,Hai->FH", G[:, o:, :o].conj(), W)
    U = x["U"] / torch.sqrt(x["V"])[:, None]
    S = ((U.conj() @ Q) * U).sum(1).real
    B = torch.from_numpy(x["basis"]).to(DEV)
    grid = torch.from_numpy(np.ascontiguousarray(x["grid"])).to(DEV)
    omega = torch.linalg.det(B).abs()
    A = torch.linalg.inv(B).T  # rows: direct coordinates
    direct = grid @ A.T
    low = torch.clamp(direct.min(0).values, max=0.0)
    high = torch.clamp(direct.max(0).values, min=0.0)
    dims = torch.floor(high - low + 1.5).long().tolist()
    origin = torch.floor(low + 0.5)
    at = torch.floor(direct + 0.5).long() - origin.long()
    box = torch.zeros(dims, device=DEV, dtype=F64)
    box[at[:, 0], at[:, 1], at[:, 2]] = S
    box = box.flatten()
    f = omega / 2.0 / math.pi ** 2
    norm = (grid ** 2).sum(1)
    keep = norm.sqrt() >= 1e-8
    low_sum = (f * S[keep] / norm[keep]).sum()
    blend = torch.tensor([[0.0, -0.5, 1.0, -0.5], [1.0, 0.0, -2.5, 1.5], [0.0, 0.5, 2.0, -1.5],
                          [0.0, 0.0, -0.5, 0.5]], device=DEV, dtype=F64)
    r = torch.arange(-N, N, device=DEV, dtype=F64) / (2.0 * N)
    shifts = torch.cartesian_prod(r, r, r) @ B
    total = torch.zeros((), device=DEV, dtype=F64)
    for part in shifts.split(max(1, 10_000_000 // grid.shape[0])):
        g = (grid[None] + part[:, None]).reshape(-1, 3)
        n2 = (g ** 2).sum(1)
        g, n2 = g[n2.sqrt() >= 1e-8], n2[n2.sqrt() >= 1e-8]
        c = g @ A.T - origin
        idx, w = [], []
        for d in range(3):
            i = c[:, d].trunc().clamp(0, dims[d] - 1)
            u = c[:, d] - i
            w.append(torch.stack([torch.ones_like(u), u, u * u, u ** 3], 1) @ blend.T)
            idx.append([(i.long() - 1 + k).clamp(0, dims[d] - 1) for k in range(4)])
        val = torch.zeros_like(n2)
        for p in range(4):
            for q in range(4):
                for s in range(4):
                    j = (idx[0][p] * dims[1] + idx[1][q]) * dims[2] + idx[2][s]
                    val += w[0][:, p] * w[1][:, q] * w[2][:, s] * box[j]
        total += (f * val / n2).sum()
    return dict(energy=torch.stack([low_sum, total / N ** 3 / 8.0]), S=S)


def exact(case, seed):
    """The outputs of run() in plain 64-bit torch (the vertex adjoint has no counterpart:
    it depends on which of the vertex blocks a formulation reads)."""
    x, kind, o = _inputs(case, seed), case["kind"], case["No"]
    x["G"] = x["G"].contiguous()
    if kind in ("ccsd", "step"):
        return _ccsd(x, case)
    if kind == "residual":
        r, R = _residual(x["t"], x["T"], x["G"], o)
        return dict(R1=r, R2=R)
    if kind == "triples":
        return _triples(x, o)
    if kind == "fsc":
        return _fsc(x, case)
    t, T = x["t"].clone().requires_grad_(), x["T"].clone().requires_grad_()
    r, R = _residual(t, T, x["G"], o)
    ((x["t_bar"] * r).sum() + (x["T_bar"] * R).sum()).backward()
    # the adjoint along symmetric amplitudes T_abij = T_baji
    return dict(T1=t.grad, T2=0.5 * (T.grad + T.grad.permute(1, 0, 3, 2)), vertex=None)
