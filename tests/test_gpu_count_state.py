"""lres_count against the state that it may not rest on or touch: trace rows exchanged after a count, and the
density array where K = Y^T Y finds no room on the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MU, E_LO = 0.02, -0.9


def _solver(precision="fp64", n=(2, 2, 2), rw=3.0):
    from lresdft_gb300 import LResGPU, system
    cr = system.jittered_h2(n, pts_per_cell=8, seed=5)
    s = LResGPU(system.LCAOBasis(cr), cr.pos, R_w=rw, M=16, precision=precision, route="tridiag", trace_rows=False)
    s.set_potential(np.linspace(-0.4, 0.1, cr.ng))
    return s


def _install(s, factor):
    """Trace rows `factor` R_W with R_W^T R_W = F_W^T F_W."""
    from lresdft_gb300 import _lib
    from lresdft_gb300.solver import trace_factor
    R = [factor * trace_factor(K) for K in s.window_blocks(s.owned_gram())]
    r_w = np.array([x.shape[0] for x in R], np.int32)
    flat = np.concatenate([x.ravel(order="F") for x in R])
    _lib.check(_lib.lib.lres_set_trace_rows(s._ctx, r_w.ctypes.data, flat.ctypes.data, None))


def test_counts_follow_the_trace_rows():
    """Rows of twice the size give four times the sums, bit for bit (every step scales by powers of two);
    without rows the counts are the owned rows' again."""
    s = _solver()
    count = lambda: np.array(s.pole_pass(MU, E_LO, want_density=False)[1:])
    own = count()
    _install(s, 1.0)
    one = count()
    _install(s, 2.0)
    assert np.array_equal(count(), 4.0 * one)
    gradient = s.adjoint(MU, E_LO)
    assert np.array_equal([gradient["N"], gradient["E"]], 4.0 * one)
    s.remove_trace_rows()
    assert np.array_equal(count(), own)
    s.close()


def test_count_without_room_leaves_the_density():
    """With 16 MB free on the device K (36 MB) does not fit: the count runs over the rows, gives the same sums (n
    roundings of 54 windows: 1e-11) and leaves the density of the last pass where it is."""
    import torch
    from lresdft_gb300.autograd import device_tensor
    warm = _solver(n=(3, 3, 3), rw=8.0)              # (every kernel loaded before the device is full)
    want = warm.pole_pass(MU + 0.05, E_LO, want_density=False)[1:]
    warm.pole_pass(MU, E_LO)
    s = _solver(n=(3, 3, 3), rw=8.0)
    dens = device_tensor(s.density_device_ptr(), s.b.cr.ng)
    s.pole_pass(MU, E_LO)
    before = dens.cpu().numpy().copy()
    torch.cuda.synchronize()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (16 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = s.pole_pass(MU + 0.05, E_LO, want_density=False)[1:]
    finally:
        del hog
        torch.cuda.empty_cache()
    assert np.array_equal(dens.cpu().numpy(), before)
    assert np.allclose(got, want, rtol=1e-11, atol=0)
    s.close()
    warm.close()
