"""Long runs of the FP32 form: the total kinetic energy against the FP64 path.
The energy weighs the distribution with v^2, so it shows what the rounding of the
last transforms and of the extracted sums adds far from the bulk of W.  Both
are done in FP64; what is left are the roundings of the FP32 sums in velocity space,
which stay where W is.  Bound: 2.5e-6, twice the FP32 unit roundoff (6e-8) times
the square root of the steps' 2 x 256 summed terms, rounded down.
"""
import numpy as np
import pytest
import torch

import orc
import qbgpu

L, R = 6.0, 3.75
BOUND = 2.5e-6


def energy(W):
    d = orc.diagnostics(W, L)
    return (d[:, 0] * (d[:, 6] + 0.5 * (d[:, 4] ** 2 + d[:, 5] ** 2))).sum()


@pytest.mark.gpu
@pytest.mark.parametrize("N,J,cells,steps,seed", [(32, 16, 8, 1000, 76), (32, 16, 8, 1000, 2), (48, 8, 4, 300, 76), (24, 8, 4, 300, 3), (64, 8, 4, 300, 76)])
def test_fp32_energy_over_long_runs(N, J, cells, steps, seed):
    q = qbgpu.Quad(N, J, J, L, R)
    h = 1.0 / cells
    W0 = torch.from_numpy(qbgpu.gaussian_mixture_state(N, L, seed=seed, ncells=cells)).cuda()
    B = torch.from_numpy(np.random.default_rng(11).standard_normal((cells, 3)) * 0.05).cuda()
    e = {}
    for prec in (64, 32):
        ws = qbgpu.Workspace(N, precision=prec)
        w, nxt = W0.clone(), torch.empty_like(W0)
        for _ in range(steps):
            qbgpu.inhom_step(ws, q, w, h, 0.4 * h / L, B, out=nxt)
            w, nxt = nxt, w
        e[prec] = energy(w.cpu().numpy())
    assert abs(e[32] - e[64]) <= BOUND * e[64], (e[32] - e[64]) / e[64]
