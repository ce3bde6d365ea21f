"""The FP32 tracer's three forms of a step (open quads, near walls and edges, decisions) at the
places where they meet: one-column-wide and tiny grids, open bottoms, isolated solid cells,
large CFL numbers, fields that are not finite.

Outcomes do not depend on which lanes share a warp, so every launch shape and claim order
gives the same particles the same ends bit for bit; against the FP64 kernel (the reference's
arithmetic) all but the few particles whose path passes within FP32 rounding of an edge agree.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 5e-9


def mask_of(kind):
    rng = np.random.default_rng(3)
    if kind == "trench":
        vac = np.zeros((24, 60), bool)
        vac[:, 44:] = True
        vac[8:16, 5:44] = True
    elif kind == "posts":            # isolated solid cells: every kind of quad
        vac = rng.random((20, 40)) > 0.12
        vac[:, 36:] = True
    elif kind == "open_bottom":      # particles leave the grid downwards and keep falling
        vac = np.ones((9, 16), bool)
        vac[3, 5:9] = False
    elif kind == "one_column":
        vac = np.ones((1, 30), bool)
        vac[:, :3] = False
    elif kind == "two_columns":
        vac = np.ones((2, 30), bool)
        vac[:, :3] = False
        vac[0, :9] = False
    else:
        vac = np.ones((3, 5), bool)  # "tiny"
        vac[1, :2] = False
    return vac


def batch(vac, n, seed, bad=None):
    rng = np.random.default_rng(seed)
    nx, ny = vac.shape
    ion = np.arange(n) < n // 2
    x = rng.uniform(0, nx * DX, n)
    y = np.full(n, (ny - 1e-3) * DX)
    vx = np.where(ion, rng.normal(0, 2e3, n), rng.normal(0, 7e5, n))
    vy = -np.where(ion, rng.uniform(5e3, 3e4, n), np.abs(rng.normal(0, 7e5, n)))
    qm = np.where(ion, 2.4e6, -1.76e11)
    spc = np.where(ion, 0, 1).astype(np.int8)
    ex, ey = rng.normal(0, 3e6, (2, nx, ny))
    if bad is not None:
        ex[nx // 2, ny // 2] = bad
    return (x, y, vx, vy, qm, spc), ex, ey


def trace(vac, parts, ex, ey, cfl, tapered, barrier, precision, shape=(0, 1), order=0, max_steps=400):
    import torch
    from trench_b200 import _capi
    from trench_b200.tracer import Context, _ptr
    L = _capi.lib()
    ctx = Context(vac, 0, DX)
    f = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    X = [f(a) for a in parts]
    EX, EY = f(ex), f(ey)
    nx, ny = vac.shape
    n = len(parts[0])
    phi, wf = None, None
    if barrier:
        rng = np.random.default_rng(9)
        phi, wf = f(rng.normal(0, 5.0, (nx, ny))), f(np.full((nx, ny), 0.8))
    ctx.check(L.tb_set_tuning(ctx.handle, *shape))
    ctx.check(L.tb_set_claim_order(ctx.handle, order))
    ctx.check(L.tb_set_fields(ctx.handle, _ptr(EX), _ptr(EY), _ptr(phi), _ptr(wf), 1e5, None))
    a = _capi.TraceArgs()
    a.n, a.max_steps, a.step_budget, a.cfl, a.tapered = n, max_steps, max_steps, cfl, int(tapered)
    a.d_x, a.d_y, a.d_vx, a.d_vy, a.d_qm, a.d_spc = (_ptr(t) for t in X)
    a.d_ex, a.d_ey, a.d_phi, a.d_wface = _ptr(EX), _ptr(EY), _ptr(phi), _ptr(wf)
    counts = torch.zeros((2, nx, ny), dtype=torch.int32, device="cuda")
    totals = torch.zeros(8, dtype=torch.int64, device="cuda")
    status = torch.full((n,), 3, dtype=torch.int8, device="cuda")
    hit = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    steps = torch.zeros(n, dtype=torch.int32, device="cuda")
    a.d_counts, a.d_totals = _ptr(counts), _ptr(totals)
    a.d_status, a.d_hit, a.d_steps = _ptr(status), _ptr(hit), _ptr(steps)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ctx.check(L.tb_trace(ctx.handle, ctypes.byref(a), _capi.PRECISION[precision], s))
    ctx.check(L.tb_check(ctx.handle, s))
    y = X[1].cpu().numpy()
    ctx.close()
    return dict(status=status.cpu().numpy(), hit=hit.cpu().numpy(), steps=steps.cpu().numpy(),
                counts=counts.cpu().numpy(), totals=totals.cpu().numpy()[:6], y=y)


@pytest.mark.parametrize("kind", ["trench", "posts", "open_bottom", "one_column", "two_columns", "tiny"])
@pytest.mark.parametrize("cfl,tapered,barrier", [(0.35, True, True), (0.35, False, False), (0.45, True, False),
                                                 (0.9, True, True)])
def test_every_form_and_launch_shape_agrees(cuda_device, kind, cfl, tapered, barrier):
    vac = mask_of(kind)
    parts, ex, ey = batch(vac, 4001, 11)
    args = (vac, parts, ex, ey, cfl, tapered, barrier)
    want = trace(*args, "f64")
    got = trace(*args, "f32")
    same = (got["status"] == want["status"]) & (got["hit"] == want["hit"])
    # about 1e-5 of the paths pass within rounding of an edge in smooth fields; this field is noise
    # from cell to cell, so paths that wander for hundreds of steps part sooner
    assert same.mean() > 0.97
    done = got["status"] != 3
    assert got["totals"][[0, 1, 2, 4, 5]].sum() == len(parts[0])
    assert (got["steps"][~done] == 400).all()
    if kind == "open_bottom":      # particles below the grid keep their distance
        below = (got["status"] == 3) & (want["status"] == 3) & (want["y"] < -20 * DX)
        assert below.sum() > 100
        # the row is an integer, so 400 steps of 2^-24 cells' rounding are next to nothing; the paths
        # that parted in the noisy field above (their velocities by up to 1e-3) and below it aside
        assert np.isclose(got["y"][below], want["y"][below], rtol=1e-3, atol=0).mean() > 0.97
    for shape, order in (((128, 1), 1), ((1024, 1), 2), ((512, 2), 0)):
        other = trace(*args, "f32", shape, order)
        for k in ("status", "hit", "steps", "counts", "totals"):
            np.testing.assert_array_equal(other[k], got[k])


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e300])
def test_fields_that_are_not_finite_stay_in_the_grid(cuda_device, bad):
    """Particles that meet a field that is not finite stop where they are until their step cap
    (counted as lost); every other particle is traced as without it."""
    vac = mask_of("trench")
    parts, ex, ey = batch(vac, 4001, 12, bad)
    got = trace(vac, parts, ex, ey, 0.35, True, True, "f32")
    assert got["totals"][[0, 1, 2, 4, 5]].sum() == len(parts[0])
    clean = trace(vac, *batch(vac, 4001, 12)[:1], *batch(vac, 4001, 12)[1:], 0.35, True, True, "f32")
    same = (got["status"] == clean["status"]) & (got["hit"] == clean["hit"])
    assert same.mean() > 0.8
    assert (got["status"][~same] == 3).all() and (got["steps"][~same] == 400).all()
