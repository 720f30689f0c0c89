"""FP64 passes on both sides of the lines that choose between the rows and the pole-weighted matrix (densities) and
between the rows and K = Y^T Y (counts), against the dense LDL^T route.  Both routes carry the rounding of
n <= 160 FP64 steps at a condition below 1e3 of z - T: n 2^-53 1e3 = 2e-11 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rw,trace", [((3, 3, 3), 1.2, True), ((3, 3, 3), 3.0, True), ((2, 2, 2), 4.6, False),
                                        ((3, 3, 3), 6.0, False), ((4, 4, 4), 1.2, True)])
@pytest.mark.parametrize("M", [4, 8, 16, 32, 64])
def test_both_sides(n, rw, trace, M):
    from lresdft_gb300 import LResGPU, system
    cr = system.jittered_h2(n, pts_per_cell=8, seed=11)
    b = system.LCAOBasis(cr, tabulation="gpu")
    v = np.linspace(-0.4, 0.1, cr.ng)
    mu, e_lo = 0.1, -1.5
    out = {}
    for route in ("ldl", "tridiag"):
        s = LResGPU(b, cr.pos, R_w=rw, M=M, precision="fp64", route=route, trace_rows=trace)
        s.set_potential(v)
        out[route] = s.pole_pass(mu, e_lo), s.pole_pass(mu, e_lo, want_density=False)[1:]
        s.close()
    (d0, N0, E0), _ = out["ldl"]
    (d1, N1, E1), (Nc, Ec) = out["tridiag"]
    assert np.max(np.abs(d1 - d0)) <= 2e-11 * np.max(np.abs(d0))
    for N, E in ((N1, E1), (Nc, Ec)):
        assert abs(N - N0) <= 2e-11 * abs(N0) and abs(E - E0) <= 2e-11 * max(abs(E0), abs(N0))
