"""Which kernels run: the I1, I2 and I4 sums at N = 32 on both sides of the rule for
the kernels of 16 values a thread (pick_chunks in csrc/qb_engine.cu, seen by the
launch accounting), and the form of the FP32 I3 sums by the state of a cell.
"""
import ctypes

import numpy as np
import pytest
import torch

import orc
import qbgpu
from conftest import rel_l1
from test_i3_pairs import states

L, R, N, J, M = 6.0, 3.75, 32, 4, 2


def launches(name):
    ms, n = ctypes.c_double(), ctypes.c_long()
    assert qbgpu.lib().qb_profile_read(name.encode(), ctypes.byref(ms), ctypes.byref(n)) == 0
    return n.value


def operators(q, prec, W):
    """Cc and Cd, and whether the wide I1 and I2 kernels ran"""
    lib = qbgpu.lib()
    lib.qb_profile_reset()
    lib.qb_profile_enable(1)
    try:
        out = qbgpu.collision_operators(qbgpu.Workspace(N, precision=prec), q, W)
        torch.cuda.synchronize()
        wide = launches("i1_terms64"), launches("i2_terms64")
        assert launches("i1_terms") == 2 and launches("i2_terms") == 1
    finally:
        lib.qb_profile_enable(0)
        lib.qb_profile_reset()
    return out, wide


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [64, 32])
def test_both_sides_of_the_wide_rule(prec):
    q = qbgpu.Quad(N, J, M, L, R)
    W = qbgpu.to_fourier(torch.from_numpy(qbgpu.gaussian_mixture_state(N, L, seed=5, ncells=8)).cuda()).repeat(80, 1, 1, 1)
    on = (2, 1) if prec == 64 else (2, 0)                # I2 in FP32 has the general kernel only
    lo, hi = 2, W.shape[0]
    assert operators(q, prec, W[:lo])[1] == (0, 0) and operators(q, prec, W[:hi])[1] == on
    while hi - lo > 1:                                   # the rule is one line in the number of cells
        n = (lo + hi) // 2
        wide = operators(q, prec, W[:n])[1]
        assert wide in ((0, 0), on)
        lo, hi = (n, hi) if wide == (0, 0) else (lo, n)
    o = orc.Oracle(N, J, M, L, R)
    w = W[1].cpu().numpy()
    for n in (lo, hi):
        (cc, cd), _ = operators(q, prec, W[:n])
        for got, want in ((cc, o.cc(w)), (cd, o.cd(w))):
            for i in (1, n - (n - 2) % 8 - 1):           # the same state, near the start and the end
                g = got[i].cpu().numpy()
                if prec == 64:
                    assert rel_l1(g, want) < 1e-12
                else:
                    assert np.linalg.norm(g - want) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.gpu
@pytest.mark.parametrize("n,real", [(8, False), (16, False), (24, True), (32, True), (48, True), (64, True), (96, True)])
def test_form_of_the_fp32_sums(n, real):
    W = np.concatenate([states(n, 1, "noise", 12), states(n, 2, "smooth", 13)])
    q, ws = qbgpu.Quad(n, 2, 3, L, R), qbgpu.Workspace(n, precision=32)
    qbgpu.collision_operators(ws, q, torch.from_numpy(W).cuda())
    assert ws.i3_forms() == ((2, 3) if real else (0, 0))
