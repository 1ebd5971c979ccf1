"""A batch captured into a CUDA graph after a larger one of the same workspace: its
scratch, the buffers of the summed partials among it, lies in that of the larger
one (summed_cells in csrc/qb_engine.cu), and its side streams exist, so nothing is
allocated while the stream is being captured.  The replay equals a direct call.
"""
import pytest
import torch

import qbgpu

L, R, J, M = 6.0, 3.75, 8, 8


@pytest.mark.gpu
@pytest.mark.parametrize("N,prec,large,small", [(8, 64, 200, 30), (16, 64, 64, 1), (16, 32, 200, 30), (32, 64, 64, 5), (32, 32, 200, 30), (64, 64, 64, 1)])
def test_capture_after_a_larger_batch(N, prec, large, small):
    q = qbgpu.Quad(N, J, M, L, R)
    W = qbgpu.to_fourier(torch.from_numpy(qbgpu.gaussian_mixture_state(N, L, seed=3, ncells=8)).cuda()).repeat(large // 8, 1, 1, 1)
    w = W[:small].clone()
    direct = qbgpu.collision_operators(qbgpu.Workspace(N, precision=prec), q, w)
    ws = qbgpu.Workspace(N, precision=prec)
    qbgpu.collision_operators(ws, q, W)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = qbgpu.collision_operators(ws, q, w)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out[0], direct[0]) and torch.equal(out[1], direct[1])


@pytest.mark.gpu
def test_capture_fp32_surrogate_after_tensor_cores():
    """the FP32 transforms of a network that ran on the tensor cores before"""
    net = qbgpu.FNO(16, width=8, modes=4, layers=2, seed=3)
    W = torch.from_numpy(qbgpu.gaussian_mixture_state(16, L, seed=3, ncells=4)).cuda()
    direct = net.forward(W)
    net = qbgpu.FNO(16, width=8, modes=4, layers=2, seed=3)
    net.set_tensor_cores(True)
    net.forward(W)
    net.set_tensor_cores(False)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = net.forward(W)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, direct)
