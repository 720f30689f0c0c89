"""dN/dmu and dE/dmu of the mixed adjoint: small differences of large sums where mu lies in a gap, so they are
taken in 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mu", [0.02, -0.2])
@pytest.mark.parametrize("n,rw,M", [((2, 2, 2), 1.2, 2), ((2, 2, 2), 3.0, 34), ((2, 2, 2), 8.0, 64), ((3, 2, 2), 5.0, 10),
                                    ((3, 3, 3), 8.0, 64)])
def test_mixed_slopes(n, rw, M, mu):
    """Against the FP64 adjoint on the same H_W.  Both sum the same FP64 tridiagonal form's resolvents, whose terms
    are of the order of the electrons whatever mu is: n 2^-53 with n <= 324 functions and a condition of
    M / (2 R) <= 1e2 is 4e-12 of them; 1e-10 leaves a factor of 25 (FP32 sweeps would leave 1e-6)."""
    from lresdft_gb300 import LResGPU, system
    cr = system.jittered_h2(n, pts_per_cell=8, seed=4)
    b = system.LCAOBasis(cr)
    H = b.H(np.linspace(-0.3, 0.1, cr.ng)).tocsr()
    out = {}
    for precision in ("fp64", "mixed"):
        s = LResGPU(b, cr.pos, R_w=rw, M=M, precision=precision, route="tridiag", trace_rows=False)
        s.set_potential(np.zeros(cr.ng))
        s.set_windows(HW=s.flatten_windows([H[W][:, W].toarray() for W in s.ctx_windows]))
        out[precision] = s.adjoint(mu, -0.9)
        s.close()
    a, m = out["fp64"], out["mixed"]
    for k in ("N", "E", "dNdmu", "dEdmu"):
        assert abs(m[k] - a[k]) <= 1e-10 * cr.n_elec, (k, m[k], a[k])
