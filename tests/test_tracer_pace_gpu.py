"""The FP32 tracer's pace where its forms of a step have cost time: particles that wait for others, and
steps beyond the quad.  Ratios of launches on the same GPU, far from what is asserted: a lane that
waits for the drain doubles the first, a staircase decision at every diagonal move the second.
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


def test_steps_beyond_the_quad_keep_pace(cuda_device):
    """A CFL number of 0.9, where a step may end beyond its quad, against 0.45, in a tapered trench: half
    as many steps, each longer."""
    vac = np.zeros((60, 150), bool)
    vac[:, 100:] = True
    for j in range(10, 100):
        w = 8 + (j - 10) // 12
        vac[30 - w:30 + w, j] = True
    parts, ex, ey = batch(vac, 1 << 18, 6)

    def make(cfl):
        return Trace(vac, parts, ex / 30, ey / 30, cfl=cfl, max_steps=2000)

    quad, beyond = least_time(lambda: make(0.45)), least_time(lambda: make(0.9))
    assert beyond < 1.5 * quad
