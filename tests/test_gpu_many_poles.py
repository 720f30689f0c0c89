"""More poles than a pass of the tridiagonal route takes (256): such contexts take the LDL^T route, and the
tridiagonal one is refused.  Against the CPU oracle's pole route, to the 1e-10 of the other parity tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-5)])
@pytest.mark.parametrize("cells", [1, 8])
def test_more_poles_than_a_pass(cells, precision, tol):
    from lresdft_gb300 import LResGPU, _lib, system
    from oracle import lrft_oracle as orc
    cr = system.jittered_h2((2, 2, 2), pts_per_cell=6, seed=5)
    b = system.LCAOBasis(cr)
    v = np.linspace(-0.4, 0.1, cr.ng).reshape(cr.shape)
    mu, e_lo, M = 0.1, -1.5, 520
    s = LResGPU(b, cr.pos[:cells], R_w=3.0, M=M, precision=precision, trace_rows=False)
    assert s.route == "ldl"
    with pytest.raises(_lib.LResError, match="256 poles"):
        s.set_route("tridiag")
    assert s.route == "ldl"
    s.set_potential(v)
    dens, N, E = s.pole_pass(mu, e_lo)
    want, N0, E0 = orc.pole_density(b.H(v), b.S, b.Xr, s.windows, s.own, cr.ng, cr.dV, mu, e_lo, M)
    assert np.max(np.abs(dens - want)) <= tol and abs(N - N0) <= tol * N0 and abs(E - E0) <= tol * N0
    s.close()
    s = LResGPU(b, cr.pos[:cells], R_w=3.0, M=512, precision=precision, trace_rows=False, route="tridiag")
    s.set_potential(v)
    want, N0, _ = orc.pole_density(b.H(v), b.S, b.Xr, s.windows, s.own, cr.ng, cr.dV, mu, e_lo, 512)
    dens, N, _ = s.pole_pass(mu, e_lo)
    assert np.max(np.abs(dens - want)) <= tol and abs(N - N0) <= tol * N0
    s.close()
