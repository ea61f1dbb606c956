"""The one-launch allocation-free derivative at the edges of its range, against
the FP64 numpy operator: the smallest grid, the longest axes (tiles of four
pencils, three-stage plans), a tile count that is not a multiple of the tile,
and replay from a captured graph.  Tolerance: that of tests/test_zz_no_alloc.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize("shape", [(16, 16, 16), (1024, 16, 16), (16, 1024, 32), (16, 16, 1024), (98, 30, 84)])
@pytest.mark.parametrize("axis,forward,power", [(0, True, 1), (1, False, -1), (2, True, 0)])
def test_against_fp64(qvti, oracle, shape, axis, forward, power):
    import torch
    from test_gpu_derivative import _numpy_q_derivative

    spacing = (10.0, 8.0, 12.0)
    f = np.random.default_rng(sum(shape) + axis).standard_normal(shape).astype(np.float32)
    d_in = torch.from_numpy(f).cuda()
    d_out = torch.full_like(d_in, float("nan"))
    torch.cuda.synchronize()
    qvti.q_derivative_noalloc(d_in.data_ptr(), d_out.data_ptr(), shape, spacing, axis, forward, power, stream=0)
    torch.cuda.synchronize()
    want = _numpy_q_derivative(f, spacing, axis, forward, power, oracle)
    got = d_out.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got - want) <= TOL * np.linalg.norm(want)


def test_graph_replay(qvti):
    import torch

    shape, spacing = (32, 48, 40), (10.0, 10.0, 10.0)
    d_in = torch.randn(shape, device="cuda")
    d_out, want = torch.empty_like(d_in), torch.empty_like(d_in)
    qvti.q_derivative_noalloc(d_in.data_ptr(), want.data_ptr(), shape, spacing, 1, True, 1,
                              stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        qvti.q_derivative_noalloc(d_in.data_ptr(), d_out.data_ptr(), shape, spacing, 1, True, 1,
                                  stream=torch.cuda.current_stream().cuda_stream)
    d_out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(d_out, want)
