"""FP64 contexts on a device with little memory left: what the fast paths would like to have is taken as far as it
is there, and the calls still answer.  The memory is taken by one tensor; allocations that fail are ordinary
errors of the library."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MU, E_LO = 0.02, -0.9


@contextlib.contextmanager
def _free(nbytes):
    """Device memory taken up to `nbytes`."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(max(torch.cuda.mem_get_info()[0] - int(nbytes), 1), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hog
        torch.cuda.empty_cache()


def _crystal():
    from lresdft_gb300 import system
    cr = system.jittered_h2((3, 3, 3), pts_per_cell=8, seed=5)
    return system.LCAOBasis(cr), cr


def test_creation_and_passes():
    """A context of 54 windows of some 290 functions with less room than its digits' workspace (some 200 MB) would
    take at its full size: fewer windows go at a time, the results are the same bit for bit.  With less than the
    tridiagonal route's buffers need at all, the automatic choice is the other route."""
    import torch

    from lresdft_gb300 import LResGPU
    b, cr = _crystal()
    v = np.linspace(-0.4, 0.1, cr.ng)

    def make():
        s = LResGPU(b, cr.pos, R_w=8.0, M=16, precision="fp64", trace_rows=False)
        s.set_potential(v)
        return s, s.pole_pass(MU, E_LO)
    warm, want = make()                              # (kernels loaded; the set-up's own temporaries measured away)
    ldl = LResGPU(b, cr.pos, R_w=8.0, M=16, precision="fp64", trace_rows=False, route="ldl")
    ldl.set_potential(v)
    dl, Nl, El = ldl.pole_pass(MU, E_LO)
    ldl.close()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    s, _ = make()
    size = free0 - torch.cuda.mem_get_info()[0]
    s.close()
    with _free(size - (100 << 20)):
        s, got = make()
        assert s.route == "tridiag"
    assert np.array_equal(got[0], want[0]) and got[1:] == want[1:]
    s.close()
    warm.close()
    with _free(size - (255 << 20)):                  # (the tridiagonal route's least: 195 MB less; the other's: 310)
        s = LResGPU(b, cr.pos, R_w=8.0, M=16, precision="fp64", trace_rows=False)
        assert s.route == "ldl"
    s.set_potential(v)                               # (its workspace is taken by the first pass)
    dl1, Nl1, El1 = s.pole_pass(MU, E_LO)
    assert np.array_equal(dl1, dl) and (Nl1, El1) == (Nl, El)
    s.close()


def test_a_refused_context_leaves_nothing():
    """The failed allocation of one call is not the next one's error."""
    from lresdft_gb300 import LResGPU, _lib
    b, cr = _crystal()
    with _free(48 << 20):
        with pytest.raises(_lib.LResError, match="out of memory"):
            LResGPU(b, cr.pos, R_w=8.0, M=16, precision="fp64", trace_rows=False)
        owner = _lib.voronoi_owner(cr.shape, cr.cell, cr.pos)
    assert owner.size == cr.ng


def test_refused_trace_rows_leave_none():
    """Trace rows that find no room: the passes run over the owned rows, as before them."""
    from lresdft_gb300 import LResGPU, _lib
    b, cr = _crystal()
    s = LResGPU(b, cr.pos, R_w=8.0, M=16, precision="fp64", route="tridiag", trace_rows=False)
    s.set_potential(np.linspace(-0.4, 0.1, cr.ng))
    want = s.pole_pass(MU, E_LO, want_density=False)[1:]
    with _free(48 << 20):                            # (the factors take 26 MB each, four times)
        with pytest.raises(_lib.LResError, match="out of memory"):
            s.install_trace_rows()
    assert s.pole_pass(MU, E_LO, want_density=False)[1:] == want
    s.set_potential(np.linspace(-0.4, 0.1, cr.ng))
    assert s.pole_pass(MU, E_LO, want_density=False)[1:] == want
    s.close()


@pytest.mark.parametrize("free_gb", [4.45, 4.2])
def test_adjoint(free_gb):
    """The adjoint keeps 4 GB of the device free.  One window of some 600 functions and 32 poles, all pole groups at
    once, wants some 0.7 GB; with less it takes fewer groups at a time.  Gradients as with the whole device: the
    same sums in another order, 10 n u of the electrons, 1e-10; the gradients by their share of kappa, whose
    denominator dN/dmu is a difference of sums of N / R."""
    from lresdft_gb300 import LResGPU, system
    n, side = 600, 5
    pos = np.array([((np.array([i, j, k]) + 0.5) * 2.0) for i in range(side) for j in range(side)
                    for k in range(side)])[:n // 6]
    cr = system.Crystal(pos, np.ones(len(pos)), np.full(3, 2.0 * side), (5 * side,) * 3, 1.0)
    b = system.LCAOBasis(cr, rcut=1.3, atom_exps=[((2.0, 1.0, 0.5), (0.8,))] * len(pos))
    s = LResGPU(b, cr.pos[:1], R_w=1e3, M=64, precision="fp64", route="tridiag", trace_rows=True)
    s.set_potential(np.linspace(-0.4, 0.1, cr.ng))
    lam = s.min_eig(-1.0, 0.0)                       # (some tens of levels below mu)
    with _free(free_gb * 2 ** 30):
        a = s.adjoint(lam + 3.0, lam - 0.3, windows=True)
    r = LResGPU(b, cr.pos[:1], R_w=1e3, M=64, precision="fp64", route="tridiag", trace_rows=True)
    r.set_potential(np.linspace(-0.4, 0.1, cr.ng))
    w = r.adjoint(lam + 3.0, lam - 0.3, windows=True)
    assert w["N"] > 1
    for k in ("N", "E", "dNdmu", "dEdmu", "kappa"):
        assert abs(a[k] - w[k]) <= 1e-10 * abs(w["N"])
    tol = 1e-10 + 10 * n * 2.0 ** -53 * w["N"] / (1.65 * abs(w["dNdmu"]))
    for k in ("dv", "dHW", "dSW"):
        assert np.max(np.abs(a[k] - w[k])) <= tol * np.max(np.abs(w[k])), (k, tol)
    s.close()
    r.close()
