"""The FP32 tridiagonal reduction with the window on its SM (and, beyond 384 functions, its first
columns from the L2-resident copy) against LAPACK, at window sizes around the edges of its tiles:
32-column blocks, the register / shared-memory boundary at 256, the resident limit at 384.

S_W = I and a random symmetric H_W are set through lres_set_windows.  Tolerances: the computed T and
Y are those of a matrix within ||dA|| <= 4 n u ||A|| of A (u = 2^-24; n Householder steps of a few
roundings each), so a Sturm count at sigma lies between the exact counts at sigma -+ ||dA||, and with
|dr_M / dlambda| <= M / (2 R) the density moves by at most M ||dA|| / (2 R) relative to its scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n):
    """One window of n functions: atoms of six functions (and one of the remainder) on a lattice with
    supports that hardly overlap."""
    from lresdft_gb300 import system
    atoms = -(-n // 6)
    side = int(np.ceil(atoms ** (1 / 3)))
    side = max(side, 2)
    pos = [((np.array([i, j, k]) + 0.5) * 2.0) for i in range(side) for j in range(side) for k in range(side)][:atoms]
    cr = system.Crystal(np.array(pos), np.ones(atoms), np.full(3, 2.0 * side), (5 * side,) * 3, 1.0)
    six = ((2.0, 1.0, 0.5), (0.8,))
    exps = [six] * atoms
    if n % 6:
        exps[-1] = (tuple(0.4 * 2.2 ** k for k in range(n % 6)), ())
    return cr, system.LCAOBasis(cr, rcut=1.3, atom_exps=exps)


@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 64, 255, 256, 257, 287, 289, 320, 321, 383, 384, 385, 401, 470])
@pytest.mark.parametrize("config", [0, 1])
def test_reduction_sizes(n, config):
    from lresdft_gb300 import LResGPU
    cr, b = _system(n)
    assert b.nb == n
    s = LResGPU(b, cr.pos[:1], R_w=1e3, M=32, precision="mixed", route="tridiag", trace_rows=False)
    s.autotune(0.0, -1.0, config=config)
    rng = np.random.default_rng(n)
    A = rng.normal(size=(n, n)) / np.sqrt(n)
    A = 0.5 * (A + A.T) + np.diag(np.linspace(-1, 1, n))
    A = A.astype(np.float32).astype(np.float64)
    s.set_windows(HW=s.flatten_windows([A]), SW=s.flatten_windows([np.eye(n)]))
    lam, C = np.linalg.eigh(A)
    dA = 4 * n * 2.0 ** -24 * np.abs(lam).max()
    for sigma in np.linspace(lam[0] - 0.1, lam[-1] + 0.1, 41):
        got = s.inertia(float(sigma))
        assert np.sum(lam < sigma - dA) <= got <= np.sum(lam < sigma + dA), (sigma, got)
    e_lo, mu, M = lam[0] - 0.3, float(np.median(lam)) + 0.05, 32
    dens, N, E = s.pole_pass(mu, e_lo)
    R = 0.5 * (mu - e_lo)
    r = 1 / (1 + ((lam - 0.5 * (mu + e_lo)) / R) ** M)
    F = np.zeros((cr.ng, n))
    F[s.ctx_own[0]] = b.Xr[s.ctx_own[0]][:, s.ctx_windows[0]].toarray()
    Y2 = (F @ C) ** 2
    want = 2 * Y2 @ r
    scale = 2 * np.sqrt(np.sum(np.sum(Y2, axis=1) ** 2))
    assert np.linalg.norm(dens - want) <= (M * dA / (2 * R) + 1e-6) * scale
    assert abs(N - cr.dV * want.sum()) <= (M * dA / (2 * R) + 1e-6) * 2 * cr.dV * Y2.sum()
    assert abs(E - 2 * cr.dV * np.sum(Y2 @ (r * lam))) <= (M * dA / R + 1e-6) * 2 * cr.dV * Y2.sum() * (np.abs(lam).max() + 1)
    s.close()


@pytest.mark.parametrize("n", [1, 2, 5, 31, 33, 63, 64, 65, 130, 257, 300, 511, 513, 600])
def test_fp64_sizes(n):
    """The FP64 tridiagonal route (products on the tensor cores, reduction, rows, pass, count, adjoint)
    on one window against numpy, around the edges of its 32- and 64-wide tiles and the 512-term runs.
    S_W has condition ~4 and the spectrum is of order one, so every step is a backward-stable sum of
    n terms: errors of a small multiple of n u ~ 1e-13 of the result; 1e-11 leaves a factor of 100."""
    from lresdft_gb300 import LResGPU
    cr, b = _system(n)
    M = 32
    s = LResGPU(b, cr.pos[:1], R_w=1e3, M=M, precision="fp64", route="tridiag", trace_rows=False)
    rng = np.random.default_rng(n)
    Q = np.linalg.qr(rng.normal(size=(n, n)))[0]
    H = (Q * np.linspace(-1, 1, n)) @ Q.T + 0.1 * np.diag(rng.normal(size=n))
    H = 0.5 * (H + H.T)
    Q = np.linalg.qr(rng.normal(size=(n, n)))[0]
    S = (Q * np.geomspace(0.5, 2.0, n)) @ Q.T
    S = 0.5 * (S + S.T)
    s.set_windows(HW=s.flatten_windows([H]), SW=s.flatten_windows([S]))
    L = np.linalg.cholesky(S)
    A = np.linalg.solve(L, np.linalg.solve(L, H).T)
    lam, C = np.linalg.eigh(0.5 * (A + A.T))
    e_lo, mu = lam[0] - 0.3, float(np.median(lam)) + 0.05
    R = 0.5 * (mu - e_lo)
    r = 1 / (1 + ((lam - 0.5 * (mu + e_lo)) / R) ** M)
    F = np.zeros((cr.ng, n))
    F[s.ctx_own[0]] = b.Xr[s.ctx_own[0]][:, s.ctx_windows[0]].toarray()
    Y2 = (F @ np.linalg.solve(L.T, C)) ** 2
    want, N0, E0 = 2 * Y2 @ r, 2 * cr.dV * float((Y2 @ r).sum()), 2 * cr.dV * float((Y2 @ (r * lam)).sum())
    dens, N, E = s.pole_pass(mu, e_lo)
    assert np.linalg.norm(dens - want) <= 1e-11 * np.linalg.norm(2 * Y2.sum(axis=1))
    assert abs(N - N0) <= 1e-11 * abs(N0) + 1e-13 and abs(E - E0) <= 1e-11 * (abs(E0) + abs(N0))
    _, N1, E1 = s.pole_pass(mu, e_lo, want_density=False)
    assert abs(N1 - N0) <= 1e-11 * abs(N0) + 1e-13 and abs(E1 - E0) <= 1e-11 * (abs(E0) + abs(N0))
    for sigma in (e_lo, 0.5 * (lam[0] + lam[-1]), lam[-1] + 0.1):
        got = s.inertia(float(sigma))
        assert np.sum(lam < sigma - 1e-11) <= got <= np.sum(lam < sigma + 1e-11)
    if n > 1:
        z = 0.5 * (mu + e_lo) + R * np.exp(1j * np.pi * (2 * np.arange(M // 2) + 1) / M)
        wk = (z - 0.5 * (mu + e_lo)) / M
        K = F.T @ F
        a = [np.zeros((n, n)) for _ in range(3)]
        for zk, w in zip(z, wk):
            G = np.linalg.inv(zk * S - H)
            for q in range(3):
                a[q] += np.real(w * zk ** q * (G @ K @ G))
        out = s.adjoint(mu, e_lo, windows=True)
        k = out["kappa"]
        for got, ref in ((out["dHW"], a[1] - k * a[0]), (out["dSW"], -(a[2] - k * a[1]))):
            ref = 4 * cr.dV * ref
            assert np.linalg.norm(got - ref.ravel(order="F")) <= 1e-10 * np.linalg.norm(4 * cr.dV * a[0])
    s.close()
