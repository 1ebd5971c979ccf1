"""The batch tuner (autotune in csrc/qb_batch.cu) times only schedules that differ
from the default: in FP64 at N = 32 and 64 the I3 sums run as term ranges, which
the chunk multiplier of the I3 sums does not reach.  The kernels launched by a
first, tuning call against those of one step tell how many candidates ran: the
default twice, every other one twice (a warm-up and a timed step), then the step
itself.
"""
import pytest
import torch

import qbgpu

L, R = 6.0, 3.75


@pytest.mark.gpu
@pytest.mark.parametrize("N,candidates", [(64, 2), (32, 3)])        # two splits of I1, I2, I4; N = 32: I3 by chunks
def test_tuner_times_no_schedule_twice(N, candidates, monkeypatch):
    W = qbgpu.to_fourier(torch.from_numpy(qbgpu.gaussian_mixture_state(N, L, seed=1)).cuda())[0]
    count = qbgpu.lib().qb_launch_count

    def launches():
        before = count()
        qbgpu.homogeneous_batch([W.clone()], 0.01, 1, J=5, M=3, L=L, R=R)
        torch.cuda.synchronize()
        return count() - before
    monkeypatch.setenv("QB_BATCH_TUNE", "0")
    one = launches()
    monkeypatch.delenv("QB_BATCH_TUNE")
    steps = 2 + 2 * candidates + 1
    assert launches() <= (steps + 0.5) * one
    assert launches() == one                                         # tuned once
