"""Workloads of the framework, as its users call it: one SCF iteration's window solve (H(v) and a
pole pass), a whole solver call with its chemical-potential search, the band-energy gradients, and
the grid steps of the SCF loop.

A case names a crystal, the solver's settings and the call; ``prepare`` builds what a program holds
before that call (basis, solver, device potential), ``run`` makes the call, ``exact`` evaluates the
same quantities in 64 bits with plain torch: window densities by generalised eigendecomposition,
gradients by dense complex solves, the grid steps by torch's FFT.  The basis matrices X, S, T and
the window lists are inputs of the window solve and are taken as such by ``exact``.

The mixed path computes in FP32 and hands its arrays over in FP64 storage; ``run`` returns its
densities and gradients as float32, the precision that they have.
"""
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from lresdft_gb300 import LResGPU, system
from lresdft_gb300.autograd import BandEnergy
from lresdft_gb300.scf import GridOps
from lresdft_gb300.solver import solved_windows, window_setup

# chemical potential and filter edge of a converged SCF step, by family of crystal: (mu, e_lo)
STATE = {"jitter": (0.02, -0.66), "cells": (-0.08, -0.70), "amorphous": (-0.33, -2.30)}


def listed():
    return [
        # the smallest whole call: 8 molecules, every window the whole cell (one merged window)
        dict(name="density-fp64-16", call="density", family="jitter", nx=2, ny=2, nz=2, pts=8, M=64, rw=8.0, precision="fp64"),
        # the 54-electron crystal, the size of a first test or of a parameter scan
        dict(name="step-fp64-54", call="step", family="jitter", nx=3, ny=3, nz=3, pts=8, M=64, rw=8.0, precision="fp64"),
        dict(name="step-mixed-54", call="step", family="jitter", nx=3, ny=3, nz=3, pts=8, M=64, rw=8.0, precision="mixed"),
        # the double-precision path at an ordinary production size
        dict(name="step-fp64-432", call="step", family="jitter", nx=6, ny=6, nz=6, pts=8, M=64, rw=8.0, precision="fp64"),
        # the 1024-electron crystal of the benchmark: one mixed SCF iteration's window solve
        dict(name="step-mixed-1024", call="step", family="jitter", nx=8, ny=8, nz=8, pts=8, M=64, rw=8.0, precision="mixed"),
        # disordered 1024 electrons: windows of uneven size, 60^3 grid, twice the poles
        dict(name="step-mixed-amorphous", call="step", family="amorphous", nx=8, ny=8, nz=8, pts=60, M=128, rw=8.0, precision="mixed"),
        # a warm solver call of the published scaling run: one window per cell, 1000 points each
        dict(name="density-mixed-cells", call="density", family="cells", nx=8, ny=8, nz=8, pts=10, M=64, rw=12.1, precision="mixed"),
        # gradients of the band energy with respect to H_W, S_W and v at a known mu, for the SCF
        # potentials of one crystal (the window arrays' length belongs to the crystal)
        dict(name="adjoint-mixed-128", call="adjoint", family="jitter", nx=4, ny=4, nz=4, pts=8, M=64, rw=8.0, precision="mixed", crystal=0),
        # a differentiable band energy at fixed electron number, forward and backward
        dict(name="grad-fp64-54", call="grad", family="jitter", nx=3, ny=3, nz=3, pts=8, M=64, rw=8.0, precision="fp64"),
        # LDA and Hartree of one SCF iteration: the benchmark's grid and the 0.25-bohr grid
        dict(name="grid-64", call="grid", nx=64, ny=64, nz=64, dx=0.5625),
        dict(name="grid-108", call="grid", nx=108, ny=108, nz=108, dx=0.25),
        # the ionic potential of a new geometry
        dict(name="ion-1024", call="ion", family="jitter", nx=8, ny=8, nz=8, pts=8, M=2, rw=3.0, precision="mixed"),
    ]


def _cells(rng, most):
    """Three cell counts of 2 or more, their product spread over [8, most] on a log scale."""
    size = math.exp(rng.uniform(math.log(8), math.log(most + 1)))
    while True:
        edge = size ** (1 / 3)
        n = [max(2, int(round(edge * math.exp(rng.uniform(-0.35, 0.35))))) for _ in range(3)]
        if math.prod(n) <= most:
            return dict(zip(("nx", "ny", "nz"), n))


def draw(rng):
    call = rng.choices(("step", "density", "adjoint", "grad", "grid", "ion"), (50, 15, 10, 5, 12, 8))[0]
    if call == "grid":
        pts = rng.choice((8, 9, 10, 12, 18))
        while True:
            n = [pts * rng.randint(3, 12) for _ in range(3)]
            if math.prod(n) <= 108 ** 3:
                return dict(call=call, nx=n[0], ny=n[1], nz=n[2], dx=round(rng.uniform(0.25, 0.6), 4))
    if call == "ion":
        return dict(call=call, family="jitter", **_cells(rng, 512), pts=rng.choice((8, 9, 10)), M=2, rw=3.0, precision="mixed")
    if call == "grad":
        return dict(call=call, family="jitter", **_cells(rng, 27), pts=8, M=rng.choice((32, 64)), rw=round(rng.uniform(6, 8), 2), precision="fp64")
    if call == "adjoint":
        return dict(call=call, family="jitter", **_cells(rng, 64), pts=rng.choice((8, 9)), M=rng.choice((32, 64)), rw=round(rng.uniform(6, 8), 2), precision="mixed",
                    crystal=rng.randrange(1000))
    precision = rng.choice(("mixed", "mixed", "fp64"))
    # (a whole call starts from its family's state: the lowest level of a disordered cell differs too
    # much from crystal to crystal to share one)
    family = rng.choices(("jitter", "cells", "amorphous"), (60, 25, 15 if call == "step" else 0))[0]
    most = 512 if precision == "mixed" else 125
    c = dict(call=call, family=family, **_cells(rng, most if family != "cells" else most // 2))
    if family == "amorphous":
        n = max(3, round((c["nx"] * c["ny"] * c["nz"]) ** (1 / 3)))
        c.update(nx=n, ny=n, nz=n, pts=round(4.5 * n / 0.6), rw=round(rng.uniform(6, 8), 2))
    elif family == "cells":
        c.update(pts=rng.choice((9, 10)), rw=round(rng.uniform(8, 12.1), 2))
    else:
        fine = math.prod((c["nx"], c["ny"], c["nz"])) <= 27
        c.update(pts=rng.choice((8, 9, 10, 12, 18) if fine else (8, 8, 9)), rw=round(rng.uniform(5.5, 8.5), 2))
    c.update(M=rng.choice((32, 64, 64, 128)), precision=precision)
    return c


# ---------------------------------------------------------------------------- inputs

def _crystal(case, seed):
    """The crystal of a case and the centres of its windows."""
    n = (case["nx"], case["ny"], case["nz"])
    seed = case.get("crystal", seed)
    if case["family"] == "amorphous":
        cr, _ = system.amorphous_h2(nmol=n[0] ** 3, box=4.5 * n[0], seed=seed, shape=(case["pts"],) * 3)
        return cr, cr.pos
    if case["family"] == "cells":
        return system.h2_crystal(n, a=6.0, pts_per_cell=case["pts"], seed=seed), system.cell_centres(n, 6.0)
    cr = system.jittered_h2(n, pts_per_cell=case["pts"], seed=seed)
    return cr, cr.pos


def _wavevectors(shape, cell):
    return [2 * math.pi * torch.fft.fftfreq(m, float(L) / m, dtype=torch.float64, device="cuda") for m, L in zip(shape, cell)]


def _ion(cr):
    """Ionic potential on the grid, from the separable structure factor."""
    k = _wavevectors(cr.shape, cr.cell)
    pos, rc = torch.as_tensor(cr.pos, device="cuda"), torch.as_tensor(cr.atom_rc, device="cuda")
    z = torch.as_tensor(cr.Z, dtype=torch.float64, device="cuda")
    e = [torch.exp(-1j * pos[:, a, None] * k[a]) * torch.exp(-k[a] ** 2 * rc[:, None] ** 2 / 4) for a in range(3)]
    s = torch.empty(tuple(cr.shape), dtype=torch.complex128, device="cuda")
    for i in range(cr.shape[0]):
        s[i] = ((z * e[0][:, i])[:, None] * e[1]).T @ e[2]
    g2 = k[0][:, None, None] ** 2 + k[1][:, None] ** 2 + k[2] ** 2
    g2[0, 0, 0] = 1.0
    s *= -4 * math.pi / g2 / float(np.prod(cr.cell))
    s[0, 0, 0] = 0
    return torch.fft.ifftn(s).real * cr.ng


def _lda(n):
    """Slater exchange and Perdew-Zunger correlation: (exc, vxc)."""
    n = n.clamp(min=1e-14)
    rs = (3 / (4 * math.pi * n)) ** (1 / 3)
    ex = -0.75 * (3 / math.pi) ** (1 / 3) * n ** (1 / 3)
    sr, lr = rs.sqrt(), rs.log()
    den = 1 + 1.0529 * sr + 0.3334 * rs
    lo = -0.1423 / den
    vlo = lo * (1 + 7 / 6 * 1.0529 * sr + 4 / 3 * 0.3334 * rs) / den
    hi = 0.0311 * lr - 0.048 + 0.0020 * rs * lr - 0.0116 * rs
    vhi = 0.0311 * lr + (-0.048 - 0.0311 / 3) + 2 / 3 * 0.0020 * rs * lr + (2 * -0.0116 - 0.0020) / 3 * rs
    return ex + torch.where(rs >= 1, lo, hi), 4 / 3 * ex + torch.where(rs >= 1, vlo, vhi)


def _smooth(shape, rng):
    """A smooth periodic field of unit rms on the grid: a few long waves."""
    ax = [torch.arange(m, dtype=torch.float64, device="cuda") * (2 * math.pi / m) for m in shape]
    f = torch.zeros(tuple(shape), dtype=torch.float64, device="cuda")
    for _ in range(6):
        w, ph, amp = rng.integers(-3, 4, 3), rng.uniform(0, 2 * math.pi), rng.normal()
        f += amp * torch.cos(ax[0][:, None, None] * int(w[0]) + ax[1][:, None] * int(w[1]) + ax[2] * int(w[2]) + ph)
    return f / f.square().mean().sqrt().clamp(min=1e-3)


def _potential(cr, seed):
    """The local potential of an SCF iteration: ions, the exchange-correlation of the mean density
    and the slow variation that the electrons add."""
    vxc = _lda(torch.tensor([cr.n_elec / (cr.ng * cr.dV)], dtype=torch.float64))[1]
    return (_ion(cr) + float(vxc) + 0.02 * _smooth(cr.shape, np.random.default_rng([seed, 1]))).reshape(-1).contiguous()


def _density(case, seed):
    """A positive density from vacuum to the core region, with the SCF loop's floor of 1e-12."""
    rng = np.random.default_rng([seed, 2])
    f = 0.7 * _smooth((case["nx"], case["ny"], case["nz"]), rng) + 0.3 * _smooth((case["nx"], case["ny"], case["nz"]), rng)
    n = 0.03 * torch.exp(2.2 * f)
    return torch.where(f < -2.0, torch.full_like(n, 1e-12), n).reshape(-1).contiguous()


def prepare(case, seed):
    if case["call"] == "grid":
        shape = (case["nx"], case["ny"], case["nz"])
        cell = case["dx"] * np.array(shape, float)
        pos = 0.5 * cell + np.array([[0, 0, -0.7], [0, 0, 0.7]])
        cr = system.Crystal(pos, np.ones(2), cell, shape, 1.0)
        s = LResGPU(system.LCAOBasis(cr, tabulation="gpu"), cr.pos, R_w=3.0, M=2, precision="mixed")
        return dict(case=case, grid=GridOps(s), dens=_density(case, seed))
    cr, centres = _crystal(case, seed)
    s = LResGPU(system.LCAOBasis(cr, tabulation="gpu"), centres, R_w=case["rw"], M=case["M"], precision=case["precision"])
    st = dict(case=case, solver=s)
    if case["call"] == "ion":
        return dict(st, grid=GridOps(s))
    st["v"] = _potential(cr, seed)
    st["mu"], st["e_lo"] = STATE[case["family"]]
    if case["call"] == "step":
        st["dens"] = torch.empty(cr.ng, dtype=torch.float64, device="cuda")
    elif case["call"] == "adjoint":
        s.set_potential(st["v"])
        size = int(s.window_offsets[-1])
        st["grads"] = [torch.empty(k, dtype=torch.float64, device="cuda") for k in (cr.ng, size, size)]
    elif case["call"] == "grad":
        st["v"] = st["v"].reshape(cr.shape).requires_grad_()
    return st


# ---------------------------------------------------------------------------- the calls

def run(st):
    case, call = st["case"], st["case"]["call"]
    if call == "grid":
        return list(st["grid"].lda_hartree_device(st["dens"]))
    if call == "ion":
        return [st["grid"].ion_potential_device()]
    s = st["solver"]
    single = (lambda t: t.float()) if case["precision"] == "mixed" else (lambda t: t)
    if call == "step":
        s.set_potential(st["v"])
        n, e = s.pole_pass_device(st["mu"], st["e_lo"], st["dens"].data_ptr())
        return [single(st["dens"]), n, e]
    if call == "density":
        s.mu, s.e_lo = st["mu"], st["e_lo"]            # a warm step from a saved state
        dens, e, mu = s.density_device(st["v"])
        # in mixed precision mu is any value whose count is within the FP32 tolerance: in the gap,
        # where the count is nearly flat, that fixes the density and the energy but few digits of mu
        return [single(dens), e] + ([mu] if case["precision"] == "fp64" else [])
    if call == "adjoint":
        dv, dh, ds = st["grads"]
        n, e, dn, de, kappa = s.adjoint_device(st["mu"], st["e_lo"], dv.data_ptr(), dh.data_ptr(), ds.data_ptr())
        return [single(dv), single(dh), single(ds), n, e, dn, de, kappa]
    s.mu, s.e_lo = st["mu"], st["e_lo"]
    st["v"].grad = None
    energy = BandEnergy.apply(st["v"], s)
    energy.backward()
    return [energy.detach(), st["v"].grad]


# ---------------------------------------------------------------------------- work

def work(case):
    if case["call"] == "grid":
        ng = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 32.0 * ng, "flops": 2 * 5.0 * ng * math.log2(ng) + 40.0 * ng}
    mol = case["nx"] * case["ny"] * case["nz"]
    a = 6.0 if case["family"] == "cells" else 4.5
    ng = case["pts"] ** 3 * (1 if case["family"] == "amorphous" else mol)
    if case["call"] == "ion":
        # separable structure factor: a complex multiply-add per atom and wave vector
        return {"bytes": 8.0 * ng + 40.0 * mol, "flops": 8.0 * ng * 2 * mol + 5.0 * ng * math.log2(ng)}
    # a window holds the atoms within rw (6 functions each), at most the crystal's
    n = min(12.0 * mol, 12.0 * 4 / 3 * math.pi * case["rw"] ** 3 / a ** 3)
    nwin = 1 if n >= 12.0 * mol else mol if case["family"] == "cells" else 2 * mol
    m = min(ng / nwin, n) if ng / nwin > 1.5 * n and case["call"] != "step" else ng / nwin
    P = case["M"] // 2
    slots = 12.0 * mol * 4 / 3 * math.pi * 5.5 ** 3 * ng / (mol * a ** 3)     # nonzeros of X
    el = 4 if case["precision"] == "mixed" else 8
    # standard form and reduction 4/3 n^3 each, rows 2 m n^2, 20 flops per pole, row and column
    solve = nwin * (8 / 3 * n ** 3 + 2 * m * n ** 2)
    one_pass = nwin * 20.0 * P * m * n
    data = el * (slots + nwin * m * n) + 16.0 * ng
    if case["call"] in ("adjoint", "grad"):
        # per pole a complex factorisation, two substitutions and one product over the rows
        grads = nwin * P * 4 * (n ** 3 / 3 + 3 * m * n ** 2)
        out = 0 if case["call"] == "grad" else 16.0 * nwin * n ** 2
        return {"bytes": data + out, "flops": grads + (solve + 4 * one_pass if case["call"] == "grad" else 0)}
    return {"bytes": data, "flops": solve + one_pass * (4 if case["call"] == "density" else 1)}


# ---------------------------------------------------------------------------- exact values

def _windows(basis, centres, rw, v):
    """Per window: functions, owned points, dense H_W, S_W and the owned rows X[own, W]."""
    cr = basis.cr
    wins, own, _ = window_setup(basis, centres, rw)
    wins, own, _ = solved_windows(basis, wins, own)     # the order of the flat window arrays
    X = basis.Xr
    H = (basis.T + (X.T @ X.multiply(v.reshape(-1, 1))) * cr.dV).toarray()
    S = basis.S.toarray()
    return [(W, o, H[np.ix_(W, W)], S[np.ix_(W, W)], X[o][:, W].toarray()) for W, o in zip(wins, own)]


def _filter(lam, mu, e_lo, M):
    return 1 / (1 + ((lam - 0.5 * (mu + e_lo)) / (0.5 * (mu - e_lo))) ** M)


def _spectra(wins):
    """Eigenvalues of every window and the squared amplitudes of its owned points, by LAPACK, a
    window to a thread."""
    def one(w):
        H, S, F = (torch.from_numpy(np.ascontiguousarray(x)) for x in w[2:])
        L = torch.linalg.cholesky(S)
        A = torch.linalg.solve_triangular(L, torch.linalg.solve_triangular(L, H, upper=False).T, upper=False)
        lam, C = torch.linalg.eigh(0.5 * (A + A.T))
        Y = F @ torch.linalg.solve_triangular(L.T, C, upper=True)
        return lam.numpy(), (Y * Y).numpy()
    threads = torch.get_num_threads()
    torch.set_num_threads(1)
    try:
        with ThreadPoolExecutor(16) as ex:
            return list(ex.map(one, wins))
    finally:
        torch.set_num_threads(threads)


def _sums(cr, wins, spectra, mu, e_lo, M):
    """Density, electron count and band energy at (mu, e_lo)."""
    dens, e = np.zeros(cr.ng), 0.0
    for (_, o, *_), (lam, y2) in zip(wins, spectra):
        r = _filter(lam, mu, e_lo, M)
        dens[o] = 2 * (y2 @ r)
        e += 2 * cr.dV * float((y2.sum(0) * r) @ lam)
    return dens, cr.dV * float(dens.sum()), e


def _fixed_n(cr, spectra, mu0, e_lo, M):
    """mu with N(mu) = N, by bisection around mu0."""
    lam = np.concatenate([x[0] for x in spectra])
    wt = 2 * cr.dV * np.concatenate([x[1].sum(0) for x in spectra])

    def count(mu):
        return float(wt @ _filter(lam, mu, e_lo, M))

    lo, hi = mu0, mu0
    step = 0.01
    while count(lo) > cr.n_elec:
        lo, step = max(lo - step, e_lo + 1e-3), 2 * step
    step = 0.01
    while count(hi) < cr.n_elec:
        hi, step = hi + step, 2 * step
    for _ in range(80):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if count(mid) < cr.n_elec else (lo, mid)
    return 0.5 * (lo + hi)


def _gradients(basis, wins, mu, e_lo, M):
    """N, E, dN/dmu, dE/dmu and the gradients at fixed N, from dense complex solves."""
    cr = basis.cr
    c, R, P = 0.5 * (mu + e_lo), 0.5 * (mu - e_lo), M // 2
    zeta = torch.exp(1j * math.pi * (2 * torch.arange(P, dtype=torch.float64, device="cuda") + 1) / M)
    z, wk, dz = c + R * zeta, R * zeta / M, 0.5 + 0.5 * zeta
    weights = torch.stack([wk, wk * z, wk * z ** 2, wk * dz, wk * z * dz])
    N = E = dN = dE = 0.0
    acc = []
    for W, o, H, S, F in wins:
        H, S, F = (torch.as_tensor(x, device="cuda") for x in (H, S, F))
        Z = torch.linalg.solve(z[:, None, None] * S - H, F.T.to(torch.complex128).expand(P, *F.T.shape))
        q = torch.einsum("ra,kar->k", F.to(torch.complex128), Z)
        Zf = Z.permute(1, 0, 2)
        A = [((Zf * w[:, None]).reshape(len(W), -1) @ Zf.reshape(len(W), -1).T).real for w in weights]
        sc = 4 * cr.dV
        n, e = sc * float((wk * q).sum().real), sc * float((wk * z * q).sum().real)
        N, E = N + n, E + e
        # w' = w / (2R); z' w d(q)/dz = -z' w <S, Z Z^T>
        dN += n / (2 * R) - sc * float((S * A[3]).sum())
        dE += e / (2 * R) + sc * float((wk * dz * q).sum().real) - sc * float((S * A[4]).sum())
        acc.append((sc * A[0], sc * A[1], sc * A[2]))
    kappa = dE / dN
    G = torch.zeros((basis.nb, basis.nb), dtype=torch.float64, device="cuda")
    dH, dS = [], []
    for (W, *_), (a0, a1, a2) in zip(wins, acc):
        h = a1 - kappa * a0
        dH.append(h.T.reshape(-1))
        dS.append(-(a2 - kappa * a1).T.reshape(-1))
        Wd = torch.as_tensor(np.asarray(W), device="cuda")
        G[Wd[:, None], Wd[None, :]] += h
    X = basis.Xr
    XG = X @ G.cpu().numpy()
    dv = cr.dV * np.asarray(X.multiply(XG).sum(axis=1)).ravel()
    return N, E, dN, dE, kappa, dv, dH, dS


def exact(case, seed):
    if case["call"] == "grid":
        shape = (case["nx"], case["ny"], case["nz"])
        dens = _density(case, seed)
        k = _wavevectors(shape, case["dx"] * np.array(shape, float))
        g2 = k[0][:, None, None] ** 2 + k[1][:, None] ** 2 + k[2] ** 2
        g2[0, 0, 0] = math.inf
        vh = torch.fft.ifftn(4 * math.pi * torch.fft.fftn(dens.reshape(shape)) / g2).real
        return [*_lda(dens), vh.reshape(-1)]
    cr, centres = _crystal(case, seed)
    if case["call"] == "ion":
        return [_ion(cr).reshape(-1)]
    basis = system.LCAOBasis(cr, tabulation="gpu")
    mu, e_lo = STATE[case["family"]]
    M = case["M"]
    wins = _windows(basis, centres, case["rw"], _potential(cr, seed).cpu().numpy())
    if case["call"] in ("step", "density"):
        spectra = _spectra(wins)
        if case["call"] == "density":
            mu = _fixed_n(cr, spectra, mu, e_lo, M)
        dens, n, e = _sums(cr, wins, spectra, mu, e_lo, M)
        if case["call"] == "step":
            return [dens, n, e]
        return [dens.reshape(cr.shape), e] + ([mu] if case["precision"] == "fp64" else [])
    if case["call"] == "grad":
        mu = _fixed_n(cr, _spectra(wins), mu, e_lo, M)
        _, E, _, _, _, dv, _, _ = _gradients(basis, wins, mu, e_lo, M)
        return [torch.tensor(E, dtype=torch.float64), dv.reshape(cr.shape)]
    N, E, dN, dE, kappa, dv, dH, dS = _gradients(basis, wins, mu, e_lo, M)
    return [dv, torch.cat(dH), torch.cat(dS), N, E, dN, dE, kappa]
