"""The FP32 tracer has one arithmetic: a particle ends the same, bit for bit, with its field in
shared or in global memory, and a field or velocity that is not a number leaves it in its cell.

A case pack with one grid too large for shared memory traces all its cases from global memory,
where every step takes the full form; alone, the small cases take the three shared-memory forms.
"""
import ctypes

import numpy as np
import pytest

from test_tracer_forms_gpu import DX, batch, mask_of

pytestmark = pytest.mark.gpu

PERIOD = 4e-10


class Trace:
    """One case: context, fields and particles on the device."""

    def __init__(self, vac, parts, ex, ey, cfl=0.35, tapered=True, barrier=True, n_phase=0, max_steps=400, order=0):
        import torch
        from trench_b200 import _capi
        from trench_b200.tracer import Context, _ptr
        self.keep, self.vac = [], vac
        L = self.L = _capi.lib()

        def dev(a):
            self.keep.append(torch.from_numpy(np.ascontiguousarray(a)).cuda())
            return _ptr(self.keep[-1])

        def zeros(shape, dtype, fill=0):
            self.keep.append(torch.full(shape, fill, dtype=dtype, device="cuda"))
            return self.keep[-1]

        nx, ny = vac.shape
        n = len(parts[0])
        rng = np.random.default_rng(9)
        self.ctx = ctx = Context(vac, 0, DX)
        ctx.check(L.tb_set_claim_order(ctx.handle, order))
        a = self.args = _capi.TraceArgs()
        a.n, a.max_steps, a.step_budget, a.cfl, a.tapered, a.write_state = n, max_steps, max_steps, cfl, int(tapered), 1
        self.state = [torch.from_numpy(np.ascontiguousarray(p)).cuda() for p in parts]
        a.d_x, a.d_y, a.d_vx, a.d_vy, a.d_qm, a.d_spc = (_ptr(t) for t in self.state)
        a.d_ex, a.d_ey = dev(ex), dev(ey)
        if barrier:
            a.d_phi, a.d_wface = dev(rng.normal(0, 5.0, (nx, ny))), dev(np.full((nx, ny), 0.8))
        ctx.check(L.tb_set_fields(ctx.handle, a.d_ex, a.d_ey, a.d_phi, a.d_wface, 1e5, None))
        if n_phase:
            t = np.arange(n_phase) / n_phase * 2 * np.pi
            wave = np.stack([30 * np.sin(t), 10 * np.cos(t)], axis=1)
            a.d_rf_ex, a.d_rf_ey, a.d_rf_phi, a.d_wave = (
                dev(rng.normal(0, 1e5, (2, nx, ny))), dev(rng.normal(0, 1e5, (2, nx, ny))),
                dev(rng.normal(0, 0.05, (2, nx, ny))), dev(wave))
            a.n_phase, a.period, a.dt_max = n_phase, PERIOD, PERIOD / 8
            a.bound_vs, a.bound_vm = (float(v) for v in np.abs(wave).max(axis=0))
            self.clock = torch.from_numpy(np.column_stack((rng.uniform(0, PERIOD, n), np.zeros(n)))).cuda()
            a.d_clock = _ptr(self.clock)
            ctx.check(L.tb_set_rf_fields(ctx.handle, a.d_rf_ex, a.d_rf_ey, a.d_rf_phi, a.d_wface, a.d_wave, n_phase, None))
        self.counts, self.totals = zeros((2, nx, ny), torch.int32), zeros((8,), torch.int64)
        self.status, self.hit = zeros((n,), torch.int8, 3), zeros((n,), torch.int32, -1)
        self.steps = zeros((n,), torch.int32)
        a.d_counts, a.d_totals, a.d_status, a.d_hit, a.d_steps = (
            _ptr(t) for t in (self.counts, self.totals, self.status, self.hit, self.steps))

    def outcome(self):
        out = dict(counts=self.counts, totals=self.totals[:6], status=self.status, hit=self.hit, steps=self.steps)
        out.update(zip(("x", "y", "vx", "vy"), self.state))
        if self.args.n_phase:
            out["clock"] = self.clock
        return {k: v.cpu().numpy() for k, v in out.items()}

    def alone(self):
        self.ctx.check(self.L.tb_trace(self.ctx.handle, ctypes.byref(self.args), 1, None))
        self.ctx.check(self.L.tb_check(self.ctx.handle, None))
        return self.outcome()


def test_precision_code():
    from trench_b200 import _capi
    assert _capi.PRECISION["f32"] == 1


def trace_pack(cases):
    from trench_b200 import _capi
    L = cases[0].L
    pack = ctypes.c_void_p()
    handles = (ctypes.c_void_p * len(cases))(*[c.ctx.handle for c in cases])
    args = (_capi.TraceArgs * len(cases))(*[c.args for c in cases])
    assert L.tb_pack_create(ctypes.byref(pack), len(cases), handles) == 0
    assert L.tb_pack_set_args(pack, args) == 0
    assert L.tb_pack_trace(pack, 0, None) == 0
    assert L.tb_pack_check(pack, None) == 0
    L.tb_pack_destroy(pack)
    return [c.outcome() for c in cases]


def large():
    """A grid beyond shared memory (200 x 160 cells x 8 bytes) with a trench."""
    vac = np.zeros((200, 160), bool)
    vac[:, 110:] = True
    vac[60:140, 5:110] = True
    return vac


@pytest.mark.parametrize("kind", ["trench", "posts", "open_bottom", "one_column", "two_columns", "tiny"])
@pytest.mark.parametrize("cfl,tapered,barrier,n_phase", [(0.35, True, True, 0), (0.35, False, False, 0), (0.45, True, False, 0),
                                                         (0.9, True, True, 0), (0.35, True, True, 64),
                                                         (0.9, True, True, 4096)])
def test_shared_and_global_fields_give_the_same_ends(cuda_device, kind, cfl, tapered, barrier, n_phase):
    vac = mask_of(kind)
    parts, ex, ey = batch(vac, 4001, 11)
    args = (vac, parts, ex, ey, cfl, tapered, barrier, n_phase)
    want = Trace(*args).alone()
    big, parts2, ex2, ey2 = large(), *batch(large(), 501, 12)
    got = trace_pack([Trace(*args), Trace(big, parts2, ex2, ey2)])[0]
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)


def lost_in_place(vac, parts, out, clean):
    """Particles whose end the bad field changed are lost in a vacuum cell; all others end as without
    it, and the counts are those of the hits."""
    same = (out["status"] == clean["status"]) & (out["hit"] == clean["hit"]) & (out["steps"] == clean["steps"])
    assert 0 < (~same).sum() < 0.2 * len(same)
    assert (out["status"][~same] == 3).all() and (out["steps"][~same] == 400).all()
    x, y = out["x"][~same] / DX, out["y"][~same] / DX
    assert np.isfinite(x).all() and np.isfinite(y).all()
    assert vac[np.floor(x + 1e-6).astype(int) % vac.shape[0], np.floor(y).astype(int)].all()
    per_cell = np.zeros((2, vac.size), int)
    hits = out["status"] == 1
    np.add.at(per_cell, (parts[5][hits], out["hit"][hits]), 1)
    np.testing.assert_array_equal(out["counts"].reshape(2, -1), per_cell)
    assert out["totals"][[0, 1, 2, 4, 5]].sum() == len(parts[0])


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e300])
@pytest.mark.parametrize("order", [0, 2])
def test_a_field_that_is_not_finite_keeps_its_particles_in_place(cuda_device, bad, order):
    for vac in (mask_of("trench"), large()):
        parts, ex, ey = batch(vac, 4001, 12)
        clean = Trace(vac, parts, ex, ey, order=order).alone()
        ex[vac.shape[0] // 2, -6] = bad
        out = Trace(vac, parts, ex, ey, order=order).alone()
        lost_in_place(vac, parts, out, clean)


@pytest.mark.parametrize("bad", [np.nan, 1e300])
def test_a_bad_field_under_rf_stays_in_the_arrays(cuda_device, bad):
    """There a step that is not a number lasts dt_max, and its particle may leave the grid; every
    particle still ends once, and the counts are those of the hits."""
    for vac in (mask_of("trench"), large()):
        parts, ex, ey = batch(vac, 4001, 12)
        ex[vac.shape[0] // 2, -6] = bad
        out = Trace(vac, parts, ex, ey, n_phase=64).alone()
        assert out["totals"][[0, 1, 2, 4, 5]].sum() == len(parts[0])
        assert out["counts"].sum() == (out["status"] == 1).sum()


def test_a_long_fall_stays_below_the_grid(cuda_device):
    """More rows below the grid than the 16 bits that the drain keeps of a row."""
    vac = mask_of("open_bottom")
    parts, ex, ey = batch(vac, 64, 5)
    out = Trace(vac, parts, 0 * ex, 0 * ey, cfl=0.9, barrier=False, max_steps=60000).alone()
    fell = out["status"] == 3
    assert fell.any()
    # some fall steeply; the drain lets a particle fall no further than 64 steps from its last row
    assert (out["y"][fell] / DX > -33000).all() and (out["y"][fell] / DX).min() < -32768 + 1
