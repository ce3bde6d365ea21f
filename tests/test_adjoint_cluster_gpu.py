"""The adjoint sweeps in one launch and in launches, at the edges where one takes over from the other:
few and many slots (with and without the operator's rows in shared memory, shares of the slots
that are uneven or empty, 1024 slots and beyond), no feedback, modes below, at and above a warp,
more modes or batches than the reverse sweep's launch holds, both conductor kinds, with and
without leakage.
"""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(depth, modes, mask_type, mode, leak, chunks=(3, 3, 1), **more):
    """The sweeps against the FP64 recurrence differentiated by torch (sums in another order: 1e-9
    relative, as the recorded-run tests).  Returns the number of surface slots."""
    import torch
    from trench_b200 import adjoint
    from trench_b200.step import ChargingCase
    p, eE, wE, eA, wA = adjoint.adjoint_workload(n_per_batch=1 << 14)
    p = replace(p, trench_d=depth, mask_type=mask_type, field_mode=mode, sigma_s=1e-15 if leak else 0.0,
                substrate_voltage=-5.0 if mode == "fixed" else 0.0, **more)
    c = ChargingCase(p, capacity=16, max_batches=4)
    rng = np.random.default_rng(depth + modes)
    m = c.m
    cond = torch.from_numpy(c.t_sflag.cpu().numpy() & 1 != 0).cuda()
    bottom = torch.from_numpy(c.t_sflag.cpu().numpy() & 4 != 0).cuda()
    rho0 = torch.from_numpy(rng.normal(0, 1e3, m)).cuda() * ~cond
    h = adjoint.History(c, (eE, wE), (eA, wA), 1, 3, rho0, 0)
    for nb in chunks:
        t = rng.poisson(3.0, size=(nb, h.rows, m)).astype(np.int32)
        t[:, -2] = t[:, :h.ne].sum(axis=1)
        t[:, -1] = rng.poisson(0.9 * t[:, -2])
        h.chunks.append(torch.from_numpy(t).pin_memory())
    if modes:
        q, _ = np.linalg.qr(rng.standard_normal((m, modes)))
        h.basis = torch.from_numpy(q.copy()).cuda()
        scale = 1e-2 * p.dx ** 2 / c.q_macro / m
        for b in range(sum(chunks)):
            if b % 2 == 0:
                h.resp_i.append(torch.from_numpy(-scale * rng.random((m, modes))).cuda())
                h.resp_e.append(torch.from_numpy(scale * rng.random((m, modes))).cuda())
            h.resp_index.append(len(h.resp_i) - 1)
    w_rho = torch.from_numpy(rng.normal(0, 1e-3, m)).cuda()
    w_b = torch.from_numpy(rng.normal(0, 1.0, sum(chunks))).cuda()

    def leaves():
        return [torch.from_numpy(rng2.uniform(0.8, 1.2, k)).cuda().requires_grad_(True) for k in (h.ne, h.na)] + \
            [rho0.clone().requires_grad_(True)]

    rng2 = np.random.default_rng(5)
    a = leaves()
    rng2 = np.random.default_rng(5)
    o = leaves()
    rho, bot = adjoint.SurfaceCharge.apply(*a, h, bool(modes))
    ((rho * w_rho).sum() + (bot * w_b).sum()).backward()
    T = torch.cat(h.chunks).cuda().double()
    r, bots, dx2 = o[2], [], p.dx ** 2
    for b in range(sum(chunks)):
        ci = T[b, -2] + (o[0] - 1) @ T[b, :h.ne] + (o[1] - 1) @ T[b, h.ne:h.ne + h.na]
        ce = T[b, -1]
        if modes:
            i = h.resp_index[b]
            shift = h.basis.T @ (r - r.detach())
            ci, ce = ci + h.resp_i[i] @ shift, ce + h.resp_e[i] @ shift
        n = r + torch.where(cond, torch.zeros_like(ci), (ci - ce) * c.q_macro / dx2)
        if c.leak_M is not None:
            n = c.leak_M @ (n * dx2 + (c.leak_h if c.leak_h is not None else 0.0)) / dx2
        if c.driven:
            n = torch.where(cond, torch.zeros_like(n), n)
        if c.floating:
            drift = dx2 * (c.g_s * (n - r)).sum()
            x_i = c.q_macro * ci[cond].sum() / c.C_cond + drift
            x_e = c.q_macro * ce[cond].sum() / c.C_cond
            k = x_i / p.electron_temp_eV
            frac = -torch.expm1(-k) / k
            dv = -p.electron_temp_eV * torch.logaddexp(-k, torch.log(x_e / p.electron_temp_eV * frac))
            e = torch.zeros(m, dtype=torch.float64, device="cuda")
            e[c.c_slot] = 1.0
            n = n + e * (c.C_cond * (dv - drift) / dx2)
        r = n
        bots.append(ci[bottom].sum())
    ((r * w_rho).sum() + (torch.stack(bots) * w_b).sum()).backward()
    torch.testing.assert_close(rho.detach(), r.detach(), rtol=1e-9, atol=1e-9 * float(r.detach().abs().max()))
    torch.testing.assert_close(bot.detach(), torch.stack(bots).detach(), rtol=1e-12, atol=1e-9)
    for x, y in zip(a, o):
        torch.testing.assert_close(x.grad, y.grad, rtol=1e-9, atol=1e-9 * float(y.grad.abs().max()))
    return m

@pytest.mark.parametrize("depth,modes,mask_type,mode", [
    (12, 0, "conductor", "floating"), (100, 5, "conductor", "floating"), (100, 40, "dielectric", "floating"),
    (300, 3, "conductor", "floating"), (120, 33, "conductor", "fixed")])
@pytest.mark.parametrize("leak", [True, False])
def test_adjoint_sweeps_match_torch(cuda_device, depth, modes, mask_type, mode, leak):
    run(depth, modes, mask_type, mode, leak)


# 1024 slots and the next size; slots that eight CTAs share unevenly; 257 modes and 1030 batches, where
# the forward sweep is one launch and the reverse one is not
@pytest.mark.parametrize("depth,modes,chunks,more,slots", [
    (462, 3, (3, 2), {}, 1024), (463, 3, (3, 2), {}, 1026), (463, 0, (2,), {}, 1026), (30, 5, (3, 3, 1), dict(nx=61), 161),
    (100, 256, (3, 2), {}, 300), (100, 257, (3, 2), {}, 300), (12, 2, (1030,), {}, 124)])
@pytest.mark.parametrize("leak", [True, False])
def test_adjoint_sweeps_match_torch_at_the_edges(cuda_device, depth, modes, chunks, more, slots, leak):
    assert run(depth, modes, "conductor", "floating", leak, chunks, **more) == slots


def test_fewer_slots_than_ctas_in_the_last_share(cuda_device):
    """A short trench in a narrow grid: some CTAs of the cluster own no slots."""
    m = run(3, 3, "conductor", "floating", True, nx=9, trench_w=3, floor_t=1, mask_t=1, n_vac=8)
    assert m % 8 and -(-m // 8) * 7 >= m
