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
