"""The route that FP64 contexts of fewer than four windows choose: the dense factorisations where the windows are
small and their rows few (the reduction's launches and columns cost more there than all factorisations side by
side), the tridiagonal form otherwise.  Both routes move the levels by at most 4 n u ||H|| with n <= 96 and
||H|| <= 30 Ha, 1.3e-12 (1e-11 allowed), and the density by M / (2 R) <= 10 times that: 1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms,pts,cells,M,route", [(4, 5, 3, 32, "ldl"), (4, 6, 1, 32, "tridiag"), (8, 5, 3, 16, "ldl"),
                                                     (8, 6, 3, 16, "tridiag"), (16, 4, 3, 32, "tridiag"), (16, 4, 3, 14, "ldl")])
def test_route(atoms, pts, cells, M, route):
    from lresdft_gb300 import LResGPU, system
    side = 2 if atoms <= 8 else 3
    pos = np.array([((np.array([i, j, k]) + 0.5) * 2.0) for i in range(side) for j in range(side)
                    for k in range(side)])[:atoms]
    cr = system.Crystal(pos, np.ones(atoms), np.full(3, 2.0 * side), (pts * side,) * 3, 1.0)
    b = system.LCAOBasis(cr, rcut=1.3, atom_exps=[((2.0, 1.0, 0.5), (0.8,))] * atoms)
    out = []
    for r in ("auto", "tridiag" if route == "ldl" else "ldl"):
        s = LResGPU(b, cr.pos[:cells], R_w=1e3, M=M, precision="fp64", merge_windows=False, trace_rows=False, route=r)
        if r == "auto":
            assert s.route == route and len(s.ctx_windows) == cells
        s.set_potential(np.linspace(-0.4, 0.1, cr.ng))
        lam = s.min_eig(-1.0, 0.0)
        out.append((lam, *s.pole_pass(lam + 3.0, lam - 0.3)))
        s.close()
    (l0, d0, N0, E0), (l1, d1, N1, E1) = out
    assert N0 > 0.1 and abs(l1 - l0) <= 1e-11
    assert np.max(np.abs(d1 - d0)) <= 1e-10 * np.max(np.abs(d0)) and abs(N1 - N0) <= 1e-10 * N0 and abs(E1 - E0) <= 1e-10 * abs(E0)
