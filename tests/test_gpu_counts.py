"""Sums over G_k = (z_k - T)^-1 by blocks of 32 rows (FP64): the traces of lres_count and the pole-weighted
matrix of the density pass, against the dense LDL^T route."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [2, 10, 34])                 # 1, 5 and 17 poles: parts of the pole groups
@pytest.mark.parametrize("n,rw", [((2, 2, 2), 1.2), ((2, 2, 2), 3.0), ((2, 2, 2), 8.0), ((3, 2, 2), 4.6), ((3, 3, 3), 8.0)])
def test_blocks_of_the_resolvent(n, rw, M):
    """Windows from one molecule (less than a block) to some 300 functions (ten blocks, the last one partial).
    Both routes carry the rounding of n <= 324 FP64 steps at a condition below 1e3 of z - T: n 2^-53 1e3 =
    4e-11 relative."""
    from lresdft_gb300 import LResGPU, system
    cr = system.jittered_h2(n, pts_per_cell=8, seed=11)
    b = system.LCAOBasis(cr)
    v = np.linspace(-0.4, 0.1, cr.ng)
    mu, e_lo = 0.1, -1.5
    out = {}
    for route in ("ldl", "tridiag"):
        s = LResGPU(b, cr.pos, R_w=rw, M=M, precision="fp64", route=route, trace_rows=False)
        s.set_potential(v)
        out[route] = s.pole_pass(mu, e_lo), s.pole_pass(mu, e_lo, want_density=False)[1:]
        s.close()
    (d0, N0, E0), _ = out["ldl"]
    (d1, N1, E1), (Nc, Ec) = out["tridiag"]
    tol = 4e-11
    assert np.max(np.abs(d1 - d0)) <= tol * np.max(np.abs(d0))
    for N, E in ((N1, E1), (Nc, Ec)):
        assert abs(N - N0) <= tol * abs(N0) and abs(E - E0) <= tol * max(abs(E0), abs(N0))
