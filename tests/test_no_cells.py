"""The collision operator of no cells is refused at the fixed grid sizes (its
kernels have no empty grid) and does nothing in the any-N engine."""
import pytest
import torch

import qbgpu


@pytest.mark.gpu
@pytest.mark.parametrize("N", [8, 16, 32, 64])
def test_no_cells_are_refused(N):
    q, ws = qbgpu.Quad(N, 2, 2, 6.0, 3.75), qbgpu.Workspace(N)
    W = torch.zeros((0, 4, N, N), dtype=torch.complex128, device="cuda")
    with pytest.raises(RuntimeError):
        qbgpu.collision_operators(ws, q, W)


@pytest.mark.gpu
def test_no_cells_any_n():
    q, ws = qbgpu.Quad(24, 2, 2, 6.0, 3.75), qbgpu.Workspace(24)
    cc, cd = qbgpu.collision_operators(ws, q, torch.zeros((0, 4, 24, 24), dtype=torch.complex128, device="cuda"))
    assert cc.numel() == cd.numel() == 0
