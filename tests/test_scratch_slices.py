"""An evaluation runs over slices of its cells whose scratch keeps within a cap
(next_slice in csrc/qb_engine.cu, AnyRhs::slice in csrc/qb_anyn.cu; QB_ANYN_SLICE_MB,
4 GB by default): many slices give what one gives, and a large batch takes no more
device memory than the cap and its tables.
"""
import numpy as np
import pytest
import torch

import qbgpu
from conftest import rel_l1

L, R = 6.0, 3.75


def fourier(N, cells, seed):
    return qbgpu.to_fourier(torch.from_numpy(qbgpu.gaussian_mixture_state(N, L, seed=seed, ncells=cells)).cuda())


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("N", [8, 16, 24, 32, 64, 96])
def test_slices_give_the_same(N, prec, monkeypatch):
    """a cap of 1 MB: slices of one cell (N = 8: of a few), one with the last cells fewer"""
    cells, J, M = (37 if N == 8 else 5), 4, 3
    q, W = qbgpu.Quad(N, J, M, L, R), fourier(N, cells, 3)
    B = torch.from_numpy(np.random.default_rng(1).standard_normal((cells, 3))).cuda()
    out = []
    for mb in ("", "1"):
        monkeypatch.setenv("QB_ANYN_SLICE_MB", mb)
        ws = qbgpu.Workspace(N, precision=prec)
        out.append([*qbgpu.collision_operators(ws, q, W), qbgpu.collision_step(ws, q, W, 0.01, B)])
    for a, b in zip(*out):
        a, b = a.cpu().numpy(), b.cpu().numpy()
        for i in range(cells):                       # sums of another split: rounding of the sums alone
            assert rel_l1(b[i], a[i]) <= (1e-12 if prec == 64 else 1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("N,prec", [(16, 64), (32, 32), (48, 32)])
def test_slices_in_a_captured_step(N, prec, monkeypatch):
    """a Strang step in slices: launched, captured and replayed the same"""
    monkeypatch.setenv("QB_ANYN_SLICE_MB", "1")
    cells = 6
    q, ws = qbgpu.Quad(N, 4, 3, L, R), qbgpu.Workspace(N, precision=prec)
    W = torch.from_numpy(qbgpu.gaussian_mixture_state(N, L, seed=2, ncells=cells)).cuda()
    B = torch.zeros((cells, 3), dtype=torch.float64, device="cuda")         # one set of pointers: graphs are kept by them
    outs, out = [], torch.empty_like(W)
    for _ in range(4):
        out.zero_()
        qbgpu.inhom_step(ws, q, W, 0.1, 0.005, B, out=out)
        outs.append(out.clone())
    assert ws.graph_replays == 2
    assert all(torch.equal(o, outs[0]) for o in outs[1:])


@pytest.mark.gpu
@pytest.mark.parametrize("N,prec,cells,J,M", [(24, 64, 1500, 8, 8), (32, 32, 2048, 16, 16), (64, 32, 300, 8, 8), (64, 64, 600, 2, 2), (96, 32, 260, 2, 2)])
def test_scratch_of_large_batches(N, prec, cells, J, M):
    q, W = qbgpu.Quad(N, J, M, L, R), fourier(N, cells, 4)
    ws = qbgpu.Workspace(N, precision=prec)
    cc, cd = torch.empty_like(W), torch.empty_like(W)
    one = [x[-1].clone() for x in qbgpu.collision_operators(qbgpu.Workspace(N, precision=prec), q, W[-3:].contiguous())]
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    cc, cd = qbgpu.collision_operators(ws, q, W)
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0] - (cc.numel() + cd.numel()) * 16
    assert used <= (4096 + 256) * 2**20, used / 2**20
    for a, b in zip((cc, cd), one):
        assert rel_l1(a[-1].cpu().numpy(), b.cpu().numpy()) <= (1e-12 if prec == 64 else 1e-5)
