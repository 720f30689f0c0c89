"""The FP64 products' workspace: its address is part of a captured pass, so nothing that a context does
later may replace it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rw", [4.0, 8.0])
def test_captured_pass_survives_other_products(rw):
    """An FP64 pass captured in a CUDA graph, then a count (K = Y^T Y over many points), trace rows and an
    adjoint, then the replay: the sums of the eager pass bit for bit (no tolerance: the same kernels on the
    same operands)."""
    import torch

    from lresdft_gb300 import LResGPU, system
    cr = system.jittered_h2((2, 2, 2), pts_per_cell=14, seed=5)
    b = system.LCAOBasis(cr)
    s = LResGPU(b, cr.pos, R_w=rw, M=16, precision="fp64", route="tridiag", trace_rows=False)
    dev = torch.device("cuda", torch.cuda.current_device())
    v = torch.linspace(-0.4, 0.1, cr.ng, dtype=torch.float64, device=dev)
    mu, e_lo = 0.1, -1.5
    out = torch.zeros(2, dtype=torch.float64, device=dev)
    s.set_potential_device(v.data_ptr())
    s.pass_async(mu, e_lo, out.data_ptr())
    torch.cuda.synchronize()
    ref = out.cpu().numpy().copy()
    assert np.all(np.isfinite(ref)) and ref[0] > 0
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=side):
        st = torch.cuda.current_stream().cuda_stream
        s.set_potential_device(v.data_ptr(), st)
        s.pass_async(mu, e_lo, out.data_ptr(), st)
    N, E = s.pole_pass(mu, e_lo, want_density=False)[1:]
    assert abs(N - ref[0]) <= 1e-10 * abs(ref[0]) and abs(E - ref[1]) <= 1e-10 * abs(ref[1])
    s.adjoint(mu, e_lo)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert s.status() == 0
    assert np.array_equal(out.cpu().numpy(), ref)
    s.close()
