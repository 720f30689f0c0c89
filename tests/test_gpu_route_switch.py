"""FP64 contexts whose overlaps or trace rows change while the LDL^T route is chosen: the tridiagonal route, chosen
again, works on the new ones.  The yardstick is a context of its own that never left it: the same kernels on the
same operands, so equality bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MU, E_LO = 0.02, -0.9


def _solver(cells):
    from lresdft_gb300 import LResGPU, system
    cr = system.jittered_h2((2, 2, 2), pts_per_cell=8, seed=5)
    s = LResGPU(system.LCAOBasis(cr), cr.pos[:cells], R_w=8.0 if cells == 1 else 3.0, M=16, precision="fp64",
                route="tridiag", trace_rows=False)
    s.set_potential(np.linspace(-0.4, 0.1, cr.ng))
    return s


def _results(s):
    a = s.adjoint(MU, E_LO)
    return [*s.pole_pass(MU, E_LO), *s.pole_pass(MU, E_LO, want_density=False)[1:], a["N"], a["E"], a["dv"]]


@pytest.mark.parametrize("cells", [1, 16])
@pytest.mark.parametrize("change", ["overlaps", "rows"])
def test_changes_on_the_other_route(cells, change):
    from lresdft_gb300.autograd import window_matrices
    s, ref = _solver(cells), _solver(cells)
    SW = (1.25 * window_matrices(s)[1]).cpu().numpy()

    def apply(x):
        if change == "overlaps":
            x.set_windows(SW=SW)
        else:
            x.install_trace_rows()
    s.set_route("ldl")
    apply(s)
    s.set_route("tridiag")
    apply(ref)
    for x, y in zip(_results(s), _results(ref)):
        assert np.array_equal(x, y)
    s.close()
    ref.close()
