"""What a context keeps from the current Hamiltonian (K = Y^T Y of the FP64 counts; the potential that the mixed
adjoint assembles again) after a captured update is replayed: a replay changes the device's Hamiltonian without
running host code, so nothing may rest on a flag that only host code clears.  The yardstick is a context of its
own that gets the same Hamiltonian eagerly: the same kernels on the same operands, so equality bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MU, E_LO = 0.02, -0.9


def _solver(precision="fp64", trace_rows=False, **kw):
    from lresdft_gb300 import LResGPU, system
    cr = system.jittered_h2((2, 2, 2), pts_per_cell=8, seed=5)
    return LResGPU(system.LCAOBasis(cr), cr.pos, R_w=3.0, M=16, precision=precision, route="tridiag",
                   trace_rows=trace_rows, **kw)


def _potentials(s):
    import torch
    a = torch.linspace(-0.4, 0.1, s.b.cr.ng, dtype=torch.float64, device="cuda")
    return a, 0.8 * a.flip(0)


def _capture(calls):
    import torch
    torch.cuda.synchronize()
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=side):
        calls(torch.cuda.current_stream().cuda_stream)
    return graph


def _results(s):
    out = [s.pole_pass(MU, E_LO, want_density=False)[1:], s.window_sums()]
    a = s.adjoint(MU, E_LO, windows=True)
    return out + [a[k] for k in ("N", "E", "dNdmu", "dEdmu", "dv", "dHW", "dSW")]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("trace_rows", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sums_and_gradients_follow_a_replay(precision, trace_rows):
    import torch
    s, ref = _solver(precision, trace_rows), _solver(precision, trace_rows)
    va, vb = _potentials(s)
    v, out = va.clone(), torch.zeros(2, dtype=torch.float64, device="cuda")
    s.set_potential_device(v.data_ptr())
    s.pass_async(MU, E_LO, out.data_ptr())

    def calls(st):
        s.set_potential_device(v.data_ptr(), st)
        s.pass_async(MU, E_LO, out.data_ptr(), st)
    graph = _capture(calls)
    ref.set_potential(va)
    assert _same(_results(s), _results(ref))          # before any replay, and whatever is kept is kept now
    for new in (vb, va):
        v.copy_(new)
        graph.replay()
        torch.cuda.synchronize()
        ref.set_potential(new)
        got, want = _results(s), _results(ref)
        assert _same(got, want), (got[0], want[0])
    s.close()
    ref.close()


def test_mixed_adjoint_follows_captured_windows():
    """Window matrices set in a captured call, a potential set after the capture, then the replay: H_W is that of
    the windows again, not H(v).  And a captured potential that has not been replayed changes nothing."""
    import torch
    from lresdft_gb300.autograd import window_matrices
    s, ref = _solver("mixed"), _solver("mixed")
    va, vb = _potentials(s)
    s.set_potential(vb)
    HW = window_matrices(s)[0]
    ptr = HW.data_ptr()
    s.set_windows(HW=HW.cpu().numpy())
    from lresdft_gb300 import _lib

    def set_hw(st):
        _lib.check(_lib.lib.lres_set_windows(s._ctx, ptr, None, 1, st))
    ref.set_potential(va)
    ref.set_windows(HW=HW.cpu().numpy())
    pending = _capture(lambda st: s.set_potential_device(va.data_ptr(), st))      # (never replayed)
    assert _same(_results(s), _results(ref))
    graph = _capture(set_hw)
    s.set_potential(va)
    graph.replay()
    torch.cuda.synchronize()
    assert _same(_results(s), _results(ref))
    del pending
    s.close()
    ref.close()
