"""The surrogate's mode mixing is FP32 in both modes (include/qbgpu.h): with the
tensor cores on, a batch of 128 cells and more gives the cells what smaller batches give."""
import pytest
import torch

import qbgpu


@pytest.mark.gpu
@pytest.mark.parametrize("width,modes", [(8, 4), (32, 5)])
def test_mixing_does_not_depend_on_the_batch(width, modes):
    net = qbgpu.FNO(16, width=width, modes=modes, layers=2, seed=1)
    net.set_tensor_cores(True)
    W = torch.from_numpy(qbgpu.gaussian_mixture_state(16, 6.0, seed=2, ncells=130)).cuda()
    whole = net.forward(W)
    assert torch.equal(whole, torch.cat([net.forward(W[:65].contiguous()), net.forward(W[65:].contiguous())]))
