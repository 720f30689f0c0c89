"""Rounding of the FP64 density on the tridiagonal route against the dense factorisations', both off extended
precision on the same H_W, S_W: the two have the same bound (n u times the size of z S_W - H_W and the filter's
slope), so the tridiagonal route may be at most 3 times as far off over four crystals, in the root of the mean
square (the constants of some ten rounded products and a reduction against one elimination)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MU, E_LO, M = 0.02, -0.66, 16


def _projector(H, S):
    """Re sum_k w_k (z_k S - H)^-1 by elimination with pivoting."""
    ld, n = np.longdouble, len(H)
    H, S = H.astype(ld), S.astype(ld)
    c, R = (ld(MU) + ld(E_LO)) / 2, (ld(MU) - ld(E_LO)) / 2
    P = np.zeros((n, n), ld)
    for k in range(M // 2):
        th = ld("3.14159265358979323846264338327950288") * (2 * k + 1) / M
        zeta = np.cos(th) + 1j * np.sin(th)
        A = np.concatenate([((c + R * zeta) * S - H).astype(np.clongdouble), np.eye(n, dtype=np.clongdouble)], axis=1)
        for i in range(n):
            p = i + int(np.argmax(np.abs(A[i:, i])))
            A[[i, p]] = A[[p, i]]
            A[i] /= A[i, i]
            col = A[:, i].copy()
            col[i] = 0
            A -= np.outer(col, A[i])
        P += (R * zeta / M * A[:, n:]).real
    return P


def test_density_off_extended_precision():
    from lresdft_gb300 import LResGPU, system
    from lresdft_gb300.autograd import window_matrices
    err = {"tridiag": [], "ldl": []}
    for seed in range(4):
        cr = system.jittered_h2((2, 2, 2), pts_per_cell=8, seed=seed)
        b = system.LCAOBasis(cr, rcut=5.0)
        dens = {}
        for route in err:
            s = LResGPU(b, cr.pos[:1], R_w=1e3, M=M, precision="fp64", route=route, trace_rows=False)
            s.set_potential(np.linspace(-0.4, 0.1, cr.ng))
            dens[route] = s.pole_pass(MU, E_LO)[0]
            n = len(s.ctx_windows[0])
            H, S = (x.cpu().numpy().reshape(n, n, order="F") for x in window_matrices(s))
            F = b.Xr[:, s.ctx_windows[0]].toarray()
            s.close()
        P = _projector(0.5 * (H + H.T), 0.5 * (S + S.T))
        F = F.astype(np.longdouble)[::7]
        want = 4 * np.sum((F @ P) * F, axis=1)
        for route in err:
            d = dens[route][::7] - want
            err[route].append(float(np.sqrt(np.sum(d * d) / np.sum(want * want))))
    rms = {k: float(np.sqrt(np.mean(np.square(v)))) for k, v in err.items()}
    assert rms["tridiag"] <= 3 * rms["ldl"], err
