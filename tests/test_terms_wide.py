"""The I1, I2 and I4 sums at N = 32 on 16 values a thread (csrc/qb_terms64.cuh),
which batches large enough take: the edge of the rule, quadratures whose terms
leave a remainder over the chunks, an odd number of radial nodes.  Cc and Cd are
checked against the oracle (upstream src/integrals.c:90-379) on the first, a
middle and the last cell, with the repository's bounds: 1e-12 (relative L1) in
FP64, 1e-5 (relative L2) in FP32.
"""
import numpy as np
import pytest
import torch

import orc
import qbgpu
from conftest import rel_l1

L, R, N = 6.0, 3.75, 32
# cells x J x ceil(M / 2) pieces: beyond 8 for each of the 74 (FP64) or 148 (FP32) clusters of the I3 sums
CASES = [(16, 16, 10), (12, 7, 25), (4, 2, 300)]


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("J,M,cells", CASES)
def test_wide_terms_against_oracle(J, M, cells, prec):
    W = qbgpu.to_fourier(torch.from_numpy(qbgpu.gaussian_mixture_state(N, L, seed=5, ncells=cells)).cuda())
    cc, cd = qbgpu.collision_operators(qbgpu.Workspace(N, precision=prec), qbgpu.Quad(N, J, M, L, R), W)
    o = orc.Oracle(N, J, M, L, R)
    for i in (0, cells // 2, cells - 1):
        w = W[i].cpu().numpy()
        for got, want in ((cc[i].cpu().numpy(), o.cc(w)), (cd[i].cpu().numpy(), o.cd(w))):
            if prec == 64:
                assert rel_l1(got, want) < 1e-12
            else:
                assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
