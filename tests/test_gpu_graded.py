"""Basis functions of very different size.  D X with D = 2^d (a power of two per function) turns H, S, T into
D H D and so on, and leaves the density, N, E_band and dE/dv what they are; every step of the window solve scales
exactly, so the results are equal bit for bit.  Products that hold an operand in fixed point below its row's
largest element have to balance the terms of the sum for that."""
import copy

import numpy as np
import pytest
from scipy import sparse

pytestmark = pytest.mark.gpu

MU, E_LO = 0.02, -0.9


def _scaled(b, d):
    c = copy.copy(b)
    D = sparse.diags(np.ldexp(1.0, d))
    c.X, c.Xr = (b.X @ D).tocsc(), (b.Xr @ D).tocsr()
    c.S, c.T = (D @ b.S @ D).tocsr(), (D @ b.T @ D).tocsr()
    for A in (c.X, c.Xr, c.S, c.T):
        A.sort_indices()
    return c


def _results(b, precision, gradient):
    from lresdft_gb300 import LResGPU
    s = LResGPU(b, b.cr.pos, R_w=5.0, M=16, precision=precision, route="tridiag", trace_rows=False)
    s.set_potential(np.linspace(-0.4, 0.1, b.cr.ng))
    out = [*s.pole_pass(MU, E_LO), *s.pole_pass(MU, E_LO, want_density=False)[1:]]
    if gradient:
        a = s.adjoint(MU, E_LO, windows=True)
        W = np.concatenate([np.add.outer(b.grade[w], b.grade[w]).ravel() for w in s.ctx_windows])
        out += [a[k] for k in ("N", "E", "dNdmu", "dEdmu", "dv")] + [np.ldexp(a[k], W) for k in ("dHW", "dSW")]
    s.close()
    return out


@pytest.mark.parametrize("precision,spread,gradient", [("fp64", 40, True), ("mixed", 12, True)])
@pytest.mark.parametrize("kind", ["random", "ramp"])
def test_size_of_the_basis_functions(precision, spread, gradient, kind):
    from lresdft_gb300 import system
    cr = system.jittered_h2((3, 2, 2), pts_per_cell=8, seed=5)
    b = system.LCAOBasis(cr)
    d = np.random.default_rng(3).integers(-spread, spread + 1, b.nb) if kind == "random" else \
        np.linspace(-spread, spread, b.nb).astype(int)
    b.grade = np.zeros(b.nb, int)
    g = _scaled(b, d)
    g.grade = d
    for x, y in zip(_results(g, precision, gradient), _results(b, precision, gradient)):
        assert np.array_equal(x, y), np.max(np.abs(np.subtract(x, y))) / np.max(np.abs(y))
