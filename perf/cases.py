"""Timing cases: the calls that a user of this framework makes, over the sizes they are made at.

The main path is the energy scan (ScanSolver.solve and ScanSolver.scan): for every energy a radial sweep
whose steps invert a symmetric matrix of order N_t = (l_cont + 1)^2 + n_orb (min(l_cont, 10) + 1)^2.  The
order and the number of energies in flight set the cost of a step; the number of radial points only repeats
it, so the grids here are short and the channel sets are those of the configurations and of the tests.
Beside it: the psi sweep, the gradients (forward and reverse), the continuum-continuum dipole and the
preprocessing of a Gaussian basis.

A case's "kind" names the call; the systems are those of scatt_b200.synth.  Every grid ends at 1.4 bohr and
the energies (drawn from the seed) lie in 1.1 <= k <= 1.55: there no eigenphase of these systems comes near
pi/2, where K = tan has a pole and its rounding errors grow without bound.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "spion-emol_b200", "python"))

from scatt_b200 import _lib, adjoint, synth  # noqa: E402
from scatt_b200 import solver as S  # noqa: E402


# ---------------------------------------------------------------- the cases

R_MAX = 1.4
L_HARTREE = 8          # Hartree multipoles of a solve at l_cont 4; rounding grows as r^l beyond


def listed():
    return [
        # one energy of the H2-like system (l_cont 8, N_t 162): the smallest call, a chain of short launches
        dict(name="solve_h2_one", kind="solve", system="h2_like", l_cont=8, n_orb=1, Nr=401,
             energies=1, graphs=False),
        # the H2-like scan of 20 energies at once, chunks replayed from graphs
        dict(name="solve_h2_scan", kind="solve", system="h2_like", l_cont=8, n_orb=1, Nr=401,
             energies=20, graphs=True),
        # a quick look at a few energies of a small channel set (N_t 100)
        dict(name="solve_h2o_small", kind="solve", system="h2o_like", l_cont=4, n_orb=3, Nr=301,
             energies=3, graphs=False),
        # the channel set of the gradient configuration (l_cont 12, N_t 774), a scan of 16 energies
        dict(name="scan_h2o_l12", kind="scan", system="h2o_like", l_cont=12, n_orb=5, Nr=131,
             energies=16, slots=16, groups=2, mixed=False),
        # the benchmark's channel set (l_cont 20, N_t 1046) at one energy, as a user tries a new molecule
        dict(name="solve_h2o_l20_one", kind="solve", system="h2o_like", l_cont=20, n_orb=5, Nr=131,
             energies=1, graphs=False),
        # the same channel set as a scan with many energies in flight: the headline workload
        dict(name="scan_h2o_l20", kind="scan", system="h2o_like", l_cont=20, n_orb=5, Nr=131,
             energies=28, slots=28, groups=1, mixed=False),
        # cutoffs 10 / 13 / 16 mixed in one scan (orders 726 / 801 / 894), groups out of phase
        dict(name="scan_h2o_mixed", kind="scan", system="h2o_like", l_cont=16, n_orb=5, Nr=131,
             energies=10, slots=10, groups=2, mixed=True),
        # a larger molecule (16 centres, 9 orbitals, N_t 1314): orders beyond one block's panels
        dict(name="solve_c8f8", kind="solve", system="c8f8_like", l_cont=14, n_orb=9, Nr=131,
             energies=1, graphs=False),
        # psi(n) of two energies over the whole grid into page-locked memory (N_t 324)
        dict(name="psi_h2o", kind="psi", system="h2o_like", l_cont=8, n_orb=3, Nr=201, energies=2),
        # sigma and its gradients with respect to alpha, r_c and V(r): forward and reverse sweeps (N_t 196)
        dict(name="gradient_h2o", kind="adjoint", system="h2o_like", l_cont=6, n_orb=3, Nr=161, energies=4),
        # continuum-continuum dipoles of one final state against four intermediate states (host stacks)
        dict(name="cc_dipole_l12", kind="cc", l_cont=12, n_pts=201, n_nu=4, pol="z"),
        # a water-like basis (25 functions) expanded to l = 20 on 401 points, and its Hartree potential to l = 8
        dict(name="basis_hartree", kind="basis", Lmax=20, Nr=401, dr=0.05, n_mo=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "scan", "scan", "psi", "adjoint", "cc", "basis"])
    if kind == "solve":
        l, n_orb = rng.choice([(3, 1), (4, 3), (6, 1), (6, 2), (6, 3), (8, 1), (8, 3), (10, 3), (11, 2), (12, 5), (16, 5)])
        n_e = _log_int(rng, 1, 20 if l <= 8 else 6 if l <= 12 else 2)
        return dict(kind=kind, system="h2_like" if n_orb == 1 else "h2o_like", l_cont=l, n_orb=n_orb,
                    Nr=_log_int(rng, 131, 300 if l <= 8 else 160), energies=n_e, graphs=rng.random() < 0.5)
    if kind == "scan":
        l, n_orb, most = rng.choice([(8, 3, 32), (11, 2, 24), (12, 5, 16), (16, 5, 8), (20, 5, 8)])
        n_e = _log_int(rng, 4, most)
        return dict(kind=kind, system="h2o_like", l_cont=l, n_orb=n_orb, Nr=rng.randint(131, 145),
                    energies=n_e, slots=n_e, groups=rng.choice([1, 1, 2, 3]), mixed=rng.random() < 0.3)
    if kind == "psi":
        l, n_orb = rng.choice([(4, 3), (6, 2), (6, 3), (8, 3), (10, 3)])
        return dict(kind=kind, system="h2o_like", l_cont=l, n_orb=n_orb, Nr=rng.randint(141, 201),
                    energies=rng.randint(1, 3))
    if kind == "adjoint":
        l, n_orb = rng.choice([(4, 3), (6, 2), (6, 3)])
        return dict(kind=kind, system="h2o_like", l_cont=l, n_orb=n_orb, Nr=rng.randint(133, 165),
                    energies=rng.randint(2, 4))
    if kind == "cc":
        return dict(kind=kind, l_cont=rng.randint(3, 12), n_pts=rng.randint(51, 230), n_nu=rng.randint(1, 4),
                    pol=rng.choice("xyz"))
    return dict(kind=kind, Lmax=rng.randint(8, 24), Nr=rng.randint(201, 401), dr=rng.choice([0.02, 0.05]),
                n_mo=rng.randint(2, 7))


# ---------------------------------------------------------------- inputs

def _inputs(case):
    """The scan's energy-independent inputs, from synth (the seed draws the energies)."""
    kw = dict(Nr=case["Nr"], dr=R_MAX / (case["Nr"] - 1), l_cont=case["l_cont"])
    if case["system"] == "h2_like":
        return synth.h2_like(**kw)
    if case["system"] == "h2o_like":
        return synth.h2o_like(lmax_orb=40, n_orb=case["n_orb"], **kw)
    return synth.c8f8_like(lmax_orb=40, n_orb=case["n_orb"], Nr_store=None, **kw)


def _energies(case, seed):
    """Energies of a scan, ascending, drawn from the seed."""
    rng = np.random.default_rng(seed)
    n = case["energies"]
    k = 1.1 + 0.45 * (np.arange(n) + rng.random(n)) / n
    return 0.5 * k * k


def _cutoffs(case):
    """l_cont per energy of a mixed scan: the largest, and about 3/5 and 4/5 of it."""
    if not case["mixed"]:
        return None
    l = case["l_cont"]
    low = min(l, max(10, round(0.6 * l)))
    return [(low, max(low, round(0.8 * l)), l)[i % 3] for i in range(case["energies"])]


def _pinned(shape, dtype=np.float64):
    t = {np.dtype("f8"): torch.float64, np.dtype("i4"): torch.int32}[np.dtype(dtype)]
    return torch.zeros(shape, dtype=t, pin_memory=True).numpy()


def _shells(rng):
    """Contracted shells of a water-like molecule: O 3s 2p 1d, H 2s 1p."""
    O, H1, H2 = np.zeros(3), np.array([1.43, 0.0, 1.11]), np.array([-1.43, 0.0, 1.11])
    s = []
    for cen, ls in ((O, [0, 0, 0, 1, 1, 2]), (H1, [0, 0, 1]), (H2, [0, 0, 1])):
        top = 60.0 if cen is O else 12.0
        for i, l in enumerate(ls):
            n = 1 + (i % 3)
            s.append((cen, l, top * np.array([0.25 ** j for j in range(n)]) * 0.4 ** i * (1 + 0.1 * rng.random(n)),
                      0.4 + 0.6 * rng.random(n)))
    return s


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "cc":
        n = (case["l_cont"] + 1) ** 2
        mk = lambda *head: np.swapaxes(rng.standard_normal(head + (n, n)), -1, -2)  # noqa: E731  (column-major, as psi_sweep)
        return dict(case=case, kappa=mk(case["n_pts"]), nu=mk(case["n_nu"], case["n_pts"]))
    if kind == "basis":
        shells = _shells(rng)
        nbf = sum(2 * l + 1 for _, l, _, _ in shells)
        return dict(case=case, shells=shells, C=rng.standard_normal((case["n_mo"], nbf)) / math.sqrt(nbf),
                    occ=np.full(case["n_mo"], 2.0))
    inp = _inputs(case)
    st = dict(case=case, sol=S.ScanSolver(inp), E=_energies(case, seed))
    if kind == "solve":
        st["opts"] = S.default_opts(allow_closed_channels=1, use_graphs=1 if case["graphs"] else 0)
    elif kind == "scan":
        st["scan"] = st["sol"].scan(slots=case["slots"], groups=case["groups"], alloc=_pinned,
                                    opts=S.default_opts(allow_closed_channels=1, keep_window=0))
        st["l_cont"] = _cutoffs(case)
    elif kind == "psi":
        shape = (case["energies"], case["Nr"], st["sol"].Np, st["sol"].Np)
        st["psi"] = _pinned(shape)
        st["opts"] = S.default_opts(allow_closed_channels=1)
    else:
        st["opts"] = S.default_opts(allow_closed_channels=1)
        st["dV"] = torch.zeros(case["Nr"], st["sol"].Np, st["sol"].Np, dtype=torch.float64, device="cuda")
    return st


FIELDS = ("K_kme", "A", "B", "K_aa", "b_overlap", "D", "D_raw", "d_raw", "d_corr", "partial_sigma")


def _collect(results):
    return {f: np.concatenate([getattr(r, f).ravel() for r in results]) for f in FIELDS}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        return _collect(state["sol"].solve(state["E"], opts=state["opts"]))
    if kind == "scan":
        scan = state["scan"]
        first = scan.submit(state["E"], state["l_cont"])[0]
        got = {}
        while len(got) < len(state["E"]):
            for j, r in scan.step():
                got[j - first] = r
        return _collect([got[i] for i in range(len(got))])
    if kind == "psi":
        res, psi = state["sol"].psi_sweep(state["E"], segment=64, opts=state["opts"],
                                          alloc=lambda shape, dtype=None: state["psi"])
        return dict(psi=psi, **_collect(res))
    if kind == "adjoint":
        alpha = torch.tensor(9.6, dtype=torch.float64, requires_grad=True)
        r_c = torch.tensor(1.5, dtype=torch.float64, requires_grad=True)
        dV = state["dV"].detach().requires_grad_()
        D = adjoint.Dipoles.apply(alpha, r_c, dV, state["sol"], state["E"], 1, 64, state["opts"])
        obs = adjoint.observables(state["E"], D, -0.5)
        (obs["sigma_length_z"].sum() + obs["sigma_velocity_x"].sum()).backward()
        return dict(D=D.detach(), sigma=obs["sigma_length_z"].detach(), alpha=alpha.grad, r_c=r_c.grad, dV=dV.grad)
    if kind == "cc":
        return _lib.cc_dipole(state["kappa"], state["nu"], 0, 0.05, case["pol"])
    orb, rho = _lib.sce_basis(state["shells"], state["C"], state["occ"], case["Lmax"], case["Nr"], 0.0, case["dr"])
    return dict(orb=orb, rho=rho, V_H=_lib.hartree(rho, case["dr"], L_HARTREE))


# ---------------------------------------------------------------- what a pass cannot do without

def _sizes(case, l=None):
    l = case["l_cont"] if l is None else l
    Np = (l + 1) ** 2
    Nf = case["n_orb"] * (min(case["l_cont"], 10) + 1) ** 2
    return Np, Nf, Np + Nf


def _sweep_flops(case, l=None):
    """One energy's sweep: per radial point the symmetric inverses of S and R (n^3 each), S = A - B D^-1 B^T
    and F = B^T Sinv B (half of them, by symmetry), T = Sinv B."""
    Np, Nf, Nt = _sizes(case, l)
    return case["Nr"] * (float(Nt) ** 3 + float(Np) ** 3 + Np * Np * Nf * 3.0 + float(Np) * Nf * Nf)


def work(case):
    kind = case["kind"]
    if kind == "cc":
        n = (case["l_cont"] + 1.0) ** 2
        stacks = case["n_nu"] + 1
        return {"bytes": 8.0 * (stacks * case["n_pts"] + case["n_nu"]) * n * n,
                "flops": 2.0 * case["n_nu"] * case["n_pts"] * n ** 3}
    if kind == "basis":
        L, Nr, nf = case["Lmax"], case["Nr"], case["n_mo"] + 1
        pts = Nr * 2.0 * (L + 1) ** 2
        out = 8.0 * ((L + 1) ** 2 * nf + (L_HARTREE + 1) ** 2) * Nr
        return {"bytes": out, "flops": pts * (2.0 * 25 * case["n_mo"] + 2.0 * nf * 2 * (L + 1)) +
                nf * Nr * 2.0 * (L + 1) * (L + 1) ** 2}
    ls = _cutoffs(case) if kind == "scan" else None
    flops = sum(_sweep_flops(case, l) for l in ls) if ls else case["energies"] * _sweep_flops(case)
    Np, Nf, Nt = _sizes(case)
    nl = (case["l_cont"] + min(case["l_cont"], 10) + 1) ** 2
    ins = 8.0 * (case["n_orb"] * nl * case["Nr"] + case["Nr"])
    outs = 8.0 * case["energies"] * (4 * Np * Np + Np * (case["n_orb"] + 30))
    if kind == "psi":
        # the outer boundary value carried back: Z <- Rinv Z and the psi rows of W^-1 Z at every point
        flops += case["energies"] * case["Nr"] * 2.0 * (Nt * Nt * Np + Np * Nt * Np)
        outs += 8.0 * case["energies"] * case["Nr"] * Np * Np
    if kind == "adjoint":
        # the reverse of each inverse (two products, symmetric cotangents) and of S, T and F
        flops += case["energies"] * case["Nr"] * (3.0 * float(Nt) ** 3 + 3.0 * float(Np) ** 3 + 6.0 * Np * Np * Nf +
                                                  2.0 * Np * Nf * Nf)
        outs += 8.0 * case["Nr"] * Np * Np
    return {"bytes": ins + outs, "flops": flops}


# ---------------------------------------------------------------- 64-bit values in plain numpy

def _lm(n_l):
    return [(l, m) for l in range(n_l + 1) for m in range(-l, l + 1)]


def _legendre(n_l, x):
    """Normalised associated Legendre functions without the Condon-Shortley phase, [l][m]."""
    s = np.sqrt(np.maximum(0.0, 1.0 - x * x))
    P = {}
    for m in range(n_l + 1):
        P[m, m] = np.full_like(x, 1.0 / math.sqrt(4 * math.pi)) if m == 0 else \
            P[m - 1, m - 1] * s * math.sqrt((2.0 * m + 1) / (2.0 * m))
        for l in range(m + 1, n_l + 1):
            a = math.sqrt((4.0 * l * l - 1) / (l * l - m * m))
            b = math.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1) ** 2 - 1)) if l > m + 1 else 0.0
            P[l, m] = a * (x * P[l - 1, m] - (b * P[l - 2, m] if l > m + 1 else 0.0))
    return P


def _ylm(n_l, x, phi):
    """Real spherical harmonics at points (cos theta, phi): ((n_l + 1)^2, points)."""
    P = _legendre(n_l, x)
    return np.array([P[l, 0] if m == 0 else math.sqrt(2) * P[l, abs(m)] * (np.cos(m * phi) if m > 0 else np.sin(-m * phi))
                     for l, m in _lm(n_l)])


def _sphere(degree):
    """Points and weights that integrate products of harmonics up to this total degree."""
    x, w = np.polynomial.legendre.leggauss(degree // 2 + 1)
    n = degree + 2
    phi = 2 * math.pi * np.arange(n) / n
    return np.repeat(x, n), np.tile(phi, x.size), np.repeat(w, n) * (2 * math.pi / n)


def _exact_cc(case, seed):
    st = prepare(case, seed)
    l = case["l_cont"]
    x, phi, w = _sphere(2 * l + 2)
    Y = _ylm(l, x, phi)
    s = np.sqrt(1 - x * x)
    A = (Y * (w * {"x": s * np.cos(phi), "y": s * np.sin(phi), "z": x}[case["pol"]])) @ Y.T
    n, h = case["n_pts"], 0.05
    wt = np.zeros(n)
    m = n if n % 2 else n - 3                        # 1/3 rule, 3/8 rule on the last four points of an even count
    wt[:m] += h / 3 * np.where(np.arange(m) % 2, 4.0, 2.0)
    wt[0] -= h / 3
    wt[m - 1] -= h / 3
    if n % 2 == 0:
        wt[n - 4:] += 3 * h / 8 * np.array([1.0, 3.0, 3.0, 1.0])
    out = np.zeros((case["n_nu"],) + A.shape)
    for i in range(n):
        left = (wt[i] * h * (i + 1)) * (st["kappa"][i].T @ A)
        for v in range(case["n_nu"]):
            out[v] += left @ st["nu"][v, i]
    return out


def _exact_basis(case, seed):
    st = prepare(case, seed)
    L, Nr, dr = case["Lmax"], case["Nr"], case["dr"]
    x, w = np.polynomial.legendre.leggauss(L + 1)
    n_phi = 2 * (L + 1)
    phi = 2 * math.pi * np.arange(n_phi) / n_phi
    X, PHI = np.repeat(x, n_phi), np.tile(phi, L + 1)
    sn = np.sqrt(1 - X * X)
    dirs = np.stack([sn * np.cos(PHI), sn * np.sin(PHI), X], axis=1)
    YW = _ylm(L, X, PHI) * np.repeat(w, n_phi) * (2 * math.pi / n_phi)
    orb, rho = np.zeros((case["n_mo"], (L + 1) ** 2, Nr)), np.zeros(((L + 1) ** 2, Nr))
    for k in range(Nr):
        rows = []
        for cen, l, ex, cf in st["shells"]:
            d = k * dr * dirs - cen
            r2 = np.sum(d * d, axis=1)
            r = np.sqrt(r2)
            so = cf @ ((2 * np.sqrt(np.outer(ex, ex)) / (ex[:, None] + ex[None, :])) ** (l + 1.5)) @ cf
            dfact = math.prod(range(1, 2 * l + 2, 2))
            ct = cf / math.sqrt(so) * np.sqrt(2.0 ** (2 * l + 3.5) * ex ** (l + 1.5) / (math.sqrt(math.pi) * dfact))
            rad = np.exp(-np.outer(r2, ex)) @ ct
            Y = _ylm(l, np.where(r > 0, d[:, 2] / np.where(r > 0, r, 1.0), 1.0), np.arctan2(d[:, 1], d[:, 0]))
            ms = [0] if l == 0 else [1, -1, 0] if l == 1 else [0] + [q * m for m in range(1, l + 1) for q in (1, -1)]
            rows += [Y[l * l + l + m] * r ** l * rad for m in ms]
        psi = st["C"] @ np.array(rows)
        orb[:, :, k] = psi @ YW.T
        rho[:, k] = YW @ (st["occ"] @ (psi * psi))
    r = np.arange(Nr) * dr
    V = np.zeros(((L_HARTREE + 1) ** 2, Nr))

    def cumulative(f):
        inc = np.empty(Nr - 1)
        inc[:-1] = dr / 12 * (5 * f[:-2] + 8 * f[1:-1] - f[2:])
        inc[-1] = dr / 12 * (-f[-3] + 8 * f[-2] + 5 * f[-1])
        return np.concatenate([[0.0], np.cumsum(inc)])

    rs = np.where(r > 0, r, 1.0)
    for ch, (l, _) in enumerate(_lm(L_HARTREE)):
        if np.max(np.abs(rho[ch])) < 1e-12:
            continue
        I1 = cumulative(rho[ch] * r ** (l + 2))
        I2 = cumulative(np.where(r > 0, rho[ch] * rs ** (1 - l), 0.0))
        V[ch] = 4 * math.pi / (2 * l + 1) * (np.where(r > 0, I1 / rs ** (l + 1), 0.0) + r ** l * (I2[-1] - I2))
        if l == 0:
            V[ch, 0] = 4 * math.pi * I2[-1]
    return dict(orb=orb, rho=rho, V_H=V)


def _riccati(n_l, x):
    """x j_l(x) and x y_l(x), l <= n_l, at one x > 0 (Miller's downward and the upward recurrence)."""
    y = [-math.cos(x), -math.cos(x) / x - math.sin(x)]
    for l in range(1, n_l):
        y.append((2 * l + 1) / x * y[l] - y[l - 1])
    top = n_l + int(x) + 60
    j = np.zeros(top + 2)
    j[top] = 1e-30
    for l in range(top, 0, -1):
        j[l - 1] = (2 * l + 1) / x * j[l] - j[l + 1]
        if abs(j[l - 1]) > 1e150:
            j[l - 1:] *= 1e-150
    a, b = math.sin(x), math.sin(x) / x - math.cos(x)
    j = j * (a / j[0] if abs(j[0]) > abs(j[1]) else b / j[1])
    return j[: n_l + 1], np.array(y[: n_l + 1])


def _exact_solve(case, seed):
    """K of every energy: the Numerov ratio recurrence with the Schur complement of the exchange block."""
    inp, E = _inputs(case), _energies(case, seed)
    lc, h, Nr = case["l_cont"], inp.dr, case["Nr"]
    lx = min(lc, 10)
    n_mu, n_si, n_la = (lc + 1) ** 2, (lx + 1) ** 2, min((lc + lx + 1) ** 2, inp.Nlm_store)
    l_mu = np.array([l for l, _ in _lm(lc)])
    l_f = np.tile(np.array([l for l, _ in _lm(lx)]), inp.n_occ)
    x, phi, w = _sphere(4 * lc)
    Yb = _ylm(2 * lc, x, phi)
    Y = Yb[:n_mu]
    r = np.arange(Nr) * h
    Vs = np.zeros((Yb.shape[0], Nr))
    nH = min(Vs.shape[0], inp.V_H.shape[0])
    Vs[:nH] = inp.V_H[:nH]
    for Z, ax, ay, az in inp.atoms:
        R = math.sqrt(ax * ax + ay * ay + az * az)
        Ya = _ylm(2 * lc, np.array([az / R if R > 0 else 1.0]), np.array([math.atan2(ay, ax)]))[:, 0]
        for ch, (l, _) in enumerate(_lm(2 * lc)):
            if R > 0 or l == 0:
                with np.errstate(divide="ignore", invalid="ignore"):
                    Vs[ch] -= Z * 4 * math.pi / (2 * l + 1) * np.minimum(r, R) ** l / np.maximum(r, R) ** (l + 1) * Ya[ch]
    xx, pp, ww = _sphere(lc + 2 * lx + lc)
    YL, Yq = _ylm(lc + lx, xx, pp)[:n_la], _ylm(lc, xx, pp)
    last = np.nonzero(np.max(np.abs(inp.psi_lm[: inp.n_occ, :n_la]), axis=(0, 1)) > 1e-15)[0][-1]
    n_tr = min(Nr, int(last) + 1 + max(100, int(5.0 / h)))
    n_start = min(max(1, math.ceil(2 * math.sqrt(lx * (lx + 1) / 12))), Nr - 1)

    def V_of(n):
        if n == 0:
            return np.zeros((n_mu, n_mu))
        return (Y * (w * (Vs[:, n] @ Yb))) @ Y.T + np.diag(l_mu * (l_mu + 1.0) / (2 * r[n] ** 2))

    def shifted(M, n):
        if n >= 60:
            return M
        off = np.sum(np.abs(M), axis=1) - np.abs(np.diag(M))
        g = np.min(np.diag(M) - off)
        me = g if g > 0.051 else np.linalg.eigvalsh(M)[0]
        return M + (0.011 - me) * np.eye(n_mu) if me < 0.001 else M

    Rv = [None] * len(E)
    ks = [math.sqrt(2 * e) for e in E]
    sym = lambda M: 0.5 * (M + M.T)  # noqa: E731
    for n in range(Nr - 1):
        V, rn, rn1 = V_of(n), h * (n + 1), h * (n + 2)
        Df = np.maximum(1 - h * h / 12 * l_f * (l_f + 1.0) / rn ** 2, 0.001)
        B = None
        if 0 < n < n_tr:
            chi = (inp.psi_lm[: inp.n_occ, :n_la, n] * r[n]) @ YL
            B = np.concatenate([(Yq * (ww * c)) @ Yq[:n_si].T for c in chi], axis=1)
            B *= h * h / 12 * 2 * math.sqrt(2 * math.pi) / r[n]
        for i, e in enumerate(E):
            if n < n_start:
                d = np.zeros(n_mu + l_f.size)
                if n > 0:
                    j0, j1 = _riccati(lc, ks[i] * rn)[0], _riccati(lc, ks[i] * rn1)[0]
                    V1 = np.diag(V_of(n + 1))
                    d[:n_mu] = (1 + h * h / 6 * (e - np.diag(V))) * j0[l_mu] / ((1 + h * h / 6 * (e - V1)) * j1[l_mu])
                    Df1 = np.maximum(1 - h * h / 12 * l_f * (l_f + 1.0) / rn1 ** 2, 0.001)
                    d[n_mu:] = Df * rn ** (l_f + 1.0) / (Df1 * rn1 ** (l_f + 1.0))
                Rv[i] = np.diag(d)
                continue
            A = shifted((1 + h * h * e / 6) * np.eye(n_mu) - h * h / 6 * V, n)
            W = np.diag(np.concatenate([np.zeros(n_mu), 1 / Df]))
            if B is not None:
                Si = sym(np.linalg.inv(shifted(A - (B / Df) @ B.T, n)))
                T = Si @ (B / Df)
                W[:n_mu, n_mu:], W[n_mu:, :n_mu] = -T, -T.T
                W[n_mu:, n_mu:] += (B / Df).T @ T
            else:
                Si = sym(np.linalg.inv(A))
            W[:n_mu, :n_mu] = Si
            Rv[i] = sym(np.linalg.inv(12 * W - 10 * np.eye(W.shape[0]) - Rv[i]))
    out = []
    for i, k in enumerate(ks):
        R = np.linalg.inv(Rv[i])
        Sm = sym(R[:n_mu, :n_mu] - R[:n_mu, n_mu:] @ np.linalg.solve(R[n_mu:, n_mu:], R[n_mu:, :n_mu]))
        ra, rb = h * (Nr - 1), h * Nr
        (ja, ya), (jb, yb) = _riccati(lc, k * ra), _riccati(lc, k * rb)
        Wa = 1 + h * h / 12 * (k * k - l_mu * (l_mu + 1.0) / ra ** 2)
        Wb = 1 + h * h / 12 * (k * k - l_mu * (l_mu + 1.0) / rb ** 2)
        Km = np.linalg.solve(Sm * (Wa * ya[l_mu]) - np.diag(Wb * yb[l_mu]), np.diag(Wb * jb[l_mu]) - Sm * (Wa * ja[l_mu]))
        out.append(sym(Km).ravel())
    return dict({f: None for f in FIELDS}, K_kme=np.concatenate(out))


def exact(case, seed):
    """64-bit values without this repository's kernels.  Of a solve, K (the recurrence's own result) where the
    sweep takes numpy a few seconds; the larger sweeps take it minutes.  The wave function, the fit, the
    dipoles and the gradients follow from many more stages and have no short restatement here."""
    if case["kind"] == "cc":
        return _exact_cc(case, seed)
    if case["kind"] == "basis":
        return _exact_basis(case, seed)
    if case["kind"] == "solve" and case["system"] != "c8f8_like":
        n = _sizes(case)[2]
        if case["Nr"] * case["energies"] * (n / 160.0) ** 3 <= 2000:
            return _exact_solve(case, seed)
    return None
