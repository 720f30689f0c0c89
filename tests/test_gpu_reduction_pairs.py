"""FP64 reductions of more windows than SMs, two to an SM (windows of one size) and one to an SM (a few large windows
among small ones), against the dense LDL^T route: the rounding of n <= 360 FP64 steps at a condition below 1e3,
n 2^-53 1e3 = 4e-11 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,rw", [(160, 4.6), (157, 6.0)])
def test_against_the_factorisations(cells, rw):
    from lresdft_gb300 import LResGPU, system
    cr = system.jittered_h2((5, 4, 4), pts_per_cell=6, seed=2)
    b = system.LCAOBasis(cr, tabulation="gpu")
    centres = cr.pos[:cells].copy()
    if cells < 160:                                  # the last centres' atoms join the windows near them
        centres[8:16] = centres[:8] + 0.01
    out = []
    for route in ("ldl", "tridiag"):
        s = LResGPU(b, centres, R_w=rw, M=8, precision="fp64", route=route, trace_rows=False, merge_windows=False)
        s.set_potential(np.linspace(-0.4, 0.1, cr.ng))
        out.append((s.pole_pass(0.1, -1.5), s.ctx_nW))
        s.close()
    (d0, N0, E0), n = out[0]
    (d1, N1, E1), _ = out[1]
    assert len(n) == cells > 152 and n.max() <= 360
    assert np.max(np.abs(d1 - d0)) <= 4e-11 * np.max(np.abs(d0))
    assert abs(N1 - N0) <= 4e-11 * N0 and abs(E1 - E0) <= 4e-11 * max(abs(E0), N0)
