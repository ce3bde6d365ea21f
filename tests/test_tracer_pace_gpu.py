"""The FP32 tracer's pace where its forms of a step have cost time: particles that wait for others.
A ratio of launches on the same GPU: a block that waits for one warp before its drain doubles it.
"""
import ctypes

import numpy as np
import pytest

from test_tracer_forms_gpu import batch
from test_tracer_one_arithmetic_gpu import Trace

pytestmark = pytest.mark.gpu


def least_time(make, times=5):
    import torch
    best = float("inf")
    for _ in range(times):
        c = make()
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda.synchronize()
        a.record()
        c.ctx.check(c.L.tb_trace(c.ctx.handle, ctypes.byref(c.args), 1, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
        c.ctx.close()
    return best


def test_a_few_ended_particles_hold_no_others_up(cuda_device):
    """Most of 32 or 64 particles fall through the open bottom to their step cap: two warps take as long
    as one, also when a few lanes of the first have ended."""
    vac = np.ones((60, 120), bool)
    vac[24:36, 30:60] = False

    def make(n):
        x, y, vx, vy, qm, spc = batch(vac, 64, 1)[0]
        keep = np.r_[0:n // 2, 32:32 + n // 2]
        parts = tuple(v[keep] for v in (x, y, 0 * vx, vy, qm, spc))
        z = np.zeros(vac.shape)
        return Trace(vac, parts, z, z, barrier=False, max_steps=6000)

    one, two = least_time(lambda: make(32)), least_time(lambda: make(64))
    ended = (make(64).alone()["status"] == 1).mean()
    assert 0.05 < ended < 0.5
    assert two < 1.5 * one
