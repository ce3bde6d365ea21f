"""The work that a user of trench_b200 has it do, as cases that can be prepared, run and timed.

Each case goes through the package's public entry points: ``ChargingCase`` batches (device-drawn
or resident particles, replayed from a CUDA graph), ``ChargingBatch`` sweeps, the drop-in
``B200Tracer`` call on host arrays, the drop-in Poisson solve, a case's set-up, and the adjoint
gradient.  ``listed()`` names the cases, ``draw`` gives more of the same ranges, ``prepare`` makes
what a program holds before the call, ``run`` is one pass.  ``exact`` is the same result in 64-bit
torch without the package's code.

Counts of hits come back as floating-point tallies: a particle whose path passes within rounding
of a cell edge lands on one of two cells, so two correct tracers agree on a tally to the few
particles concerned, not on every whole number.
"""
import math
from dataclasses import replace

import numpy as np
import torch

from trench_b200 import adjoint, geometry, inject
from trench_b200.batch import ChargingBatch, sweep_params
from trench_b200.fields import FieldSolver, compute_field
from trench_b200.params import Params
from trench_b200.step import ChargingCase
from trench_b200.tracer import B200Tracer, Context

E_CHARGE, EPS0, M_E, AMU = 1.602176634e-19, 8.8541878128e-12, 9.1093837015e-31, 1.66053906660e-27
HISTORY_ROWS = 64     # history rows a case keeps; passes after that leave the history as it is


def listed():
    return [
        # The reference's CUDA benchmark batch: 60 x 200 cells, floating conductor mask, DC ions, 3000 + 3000
        # particles (the default of Params).  The smallest batch, and the one most runs take thousands of.
        dict(name="step_small", kind="step", mode="floating", nx=60, w=20, d=80, floor=10, mask=60, vac=50,
             taper=0.0, mask_taper=0.0, dielectric=False, n=3000, max_steps=3000),
        # The AR-8 charging batch of bench.py: tapered walls, dielectric mask, bimodal ion energies, 2^20 particles.
        dict(name="step_ar8", kind="step", mode="floating", nx=60, w=20, d=160, floor=10, mask=20, vac=60,
             taper=2.0, mask_taper=5.0, dielectric=True, n=1 << 19, max_steps=3000),
        # A large batch under fixed electrode voltages with driven conductors, particles resident on the device:
        # the first batch of a run, whose fields a 64-bit tracer can be held against (2^22 particles).
        dict(name="step_large_fixed", kind="step", mode="fixed", nx=60, w=20, d=160, floor=10, mask=20, vac=60,
             taper=0.0, mask_taper=0.0, dielectric=False, n=1 << 21, max_steps=3000),
        # The reference's circuit_rf benchmark batch: 120 x 560 cells, pulsed bias, 3000 + 3000 particles whose
        # longest make 10,000 steps.
        dict(name="step_rf_small", kind="step", mode="rf_pulse", nx=120, w=80, d=400, floor=50, mask=60, vac=50,
             taper=0.0, mask_taper=0.0, dielectric=False, n=3000, max_steps=10000),
        # A circuit_rf batch large enough to fill the GPU, on the AR-8 geometry with a sine bias.
        dict(name="step_rf_large", kind="step", mode="rf_sine", nx=60, w=20, d=160, floor=10, mask=20, vac=60,
             taper=0.0, mask_taper=0.0, dielectric=False, n=1 << 18, max_steps=3000),
        # A fine grid whose field does not fit in shared memory (half the resolution of bench.py's large grid).
        dict(name="step_fine", kind="step", mode="floating", nx=200, w=20, d=400, floor=10, mask=40, vac=250,
             taper=0.0, mask_taper=0.0, dielectric=True, n=1 << 18, max_steps=6000),
        # A parameter sweep: uneven cases in one launch per batch.
        dict(name="sweep", kind="sweep", cases=8, shift=0),
        # The drop-in tracer call on host arrays (the reference's CudaTracer interface), an odd count.
        dict(name="call_f32", kind="call", precision="f32", nx=60, w=20, d=160, floor=10, mask=20, vac=60,
             taper=2.0, mask_taper=5.0, dielectric=True, n=131071, max_steps=3000),
        # The reference-exact FP64 tracer: 10,000 + 10,000 particles on 80 x 110 cells (the plain method).
        dict(name="call_f64", kind="call", precision="f64", nx=80, w=20, d=60, floor=10, mask=20, vac=20,
             taper=0.0, mask_taper=0.0, dielectric=False, n=10000, max_steps=3000),
        # Setting a case up (geometry, multigrid, surface Green's operator, leakage operator).
        dict(name="setup", kind="setup", nx=60, w=20, d=160, floor=10, mask=20, vac=60, taper=2.0, mask_taper=5.0,
             dielectric=True, n=3000),
        # The drop-in Poisson solve (fields["solve"]) of one host right-hand side, floating conductor.
        dict(name="solve", kind="solve", nx=60, w=20, d=160, floor=10, mask=20, vac=60, taper=0.0, mask_taper=0.0,
             dielectric=False, rhs=1),
        # The gradient of the charging objectives over 50 recorded batches (AR 5), with field feedback.
        dict(name="adjoint", kind="adjoint", nx=60, w=20, d=100, floor=10, mask=20, vac=50, taper=0.0,
             mask_taper=0.0, dielectric=False, batches=50, modes=32),
    ]


def draw(rng):
    """One more case: the same kinds of work, sizes spread over their ranges."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("step", "step", "step", "step", "sweep", "call", "call", "setup", "solve", "adjoint"))
    if kind == "sweep":
        return dict(kind="sweep", cases=rng.randint(2, 8), shift=rng.randint(1, 1000))
    w = rng.randint(12, 32)
    c = dict(kind=kind, nx=w + rng.randint(30, 48), w=w, d=log_int(40, 180), floor=rng.randint(6, 14),
             mask=rng.randint(8, 30), vac=rng.randint(20, 70), taper=0.0, mask_taper=0.0,
             dielectric=rng.random() < 0.5)
    if rng.random() < 0.4 and w - 2 * c["d"] * math.tan(math.radians(2.0)) >= 4:
        c.update(taper=rng.uniform(0.5, 2.0), mask_taper=rng.uniform(0.0, 5.0))
    if kind == "step":
        mode = rng.choice(("floating", "floating", "fixed", "rf_sine"))
        n = log_int(3000, 1 << 18) if mode == "rf_sine" else log_int(3000, 1 << 20)
        c.update(mode=mode, n=n, max_steps=3000)
        if mode != "floating":      # electrode voltages go with a conductive mask
            c.update(dielectric=False)
    elif kind == "call":
        precision = rng.choice(("f32", "f64"))
        c.update(precision=precision, n=log_int(2000, 1 << 19 if precision == "f32" else 1 << 16), max_steps=3000)
    elif kind == "setup":
        c.update(n=3000)
    elif kind == "solve":
        c.update(rhs=rng.choice((1, 1, 3, 16)))
    else:
        c.update(batches=rng.randint(10, 60), modes=rng.choice((0, 16, 32)))
    return c


# ---- what a program holds before the call ------------------------------------------------

def params_of(case):
    mode = case.get("mode", "floating")
    p = replace(Params(), nx=case["nx"], trench_w=case["w"], trench_d=case["d"], floor_t=case["floor"],
                mask_t=case["mask"], n_vac=case["vac"], trench_taper_deg=case["taper"],
                mask_taper_deg=case["mask_taper"], mask_type="dielectric" if case["dielectric"] else "conductor",
                mask_eps_r=3.0, electron_temp_eV=3.0, n_per_batch=case.get("n", 3000),
                max_steps=case.get("max_steps", 3000), sigma_s=1e-15, field_mode="floating", bias="dc", seed=1)
    if mode == "fixed":
        p = replace(p, field_mode="fixed", substrate_voltage=-20.0, mask_voltage=-15.0)
    if mode == "rf_pulse":
        p = replace(p, field_mode="circuit_rf", bias="rf", side_bc="pillar", rf_wave="pulse", rf_freq=4e5,
                    rf_volt=5000.0, rf_duty=0.2, rf_rise=1e-8, ion_temp_eV=0.05, dt_batch=1e-4)
    if mode == "rf_sine":
        p = replace(p, field_mode="circuit_rf", bias="rf", rf_freq=13.56e6)
    if case["nx"] == 200:
        p = replace(p, dx=2.5e-9)
    return p


def circuit_of(case):
    """One period of the electrode voltages: a pulse with its 10 ns edges, or a sine."""
    mode = case.get("mode")
    if mode == "rf_pulse":
        period, k = 2.5e-6, 4096
        t = np.arange(k) * period / k
        rise, on = 1e-8, 0.2 * period
        shape = np.clip(t / rise, 0, 1) - np.clip((t - on) / rise, 0, 1)
        up = 14.0 + 90.0 * np.exp(-((t - on - rise) / 4e-8) ** 2)
        uw = -4900.0 * shape * (1.0 - 0.1 * t / period)
        return dict(t=t, uw=uw, um=uw * 0.999, up=up, V1=up - uw * 0.999)
    if mode == "rf_sine":
        period, k = 1.0 / 13.56e6, 512
        t = np.arange(k) * period / k
        s = np.sin(2 * np.pi * t / period)
        up = 12.0 + 8.0 * np.maximum(s, 0.0)
        return dict(t=t, uw=-60.0 + 70.0 * s, um=-58.0 + 66.0 * s, up=up, V1=up + 58.0 - 66.0 * s)
    return None


def energy_table():
    return inject.table_from_pdf(inject.bimodal_gaussian_pdf(40.0, 6.0, 140.0, 6.0), 1.0, 250.0)


def angle_table():
    return inject.table_from_pdf(inject.half_gaussian_pdf(math.radians(3.0)), 0.0, math.radians(20.0))


def particles(p, ny, n, seed):
    """n ions (bimodal energies, half-Gaussian angles) and n flux-Maxwellian electrons on the device."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    f = dict(dtype=torch.float64, device="cuda", generator=g)
    mass = p.ion_mass_amu * AMU
    mean = torch.where(torch.rand(n, **f) < 0.5, 40.0, 140.0)
    energy = (mean + 6.0 * torch.randn(n, **f)).clamp(min=0.0)
    theta = math.radians(3.0) * torch.randn(n, **f)
    v = torch.sqrt(2 * energy * E_CHARGE / mass)
    s = math.sqrt(p.electron_temp_eV * E_CHARGE / M_E)
    x = torch.rand(2 * n, **f) * (p.nx * p.dx)
    y = torch.full((2 * n,), (ny - 1e-3) * p.dx, dtype=torch.float64, device="cuda")
    vx = torch.cat([v * torch.sin(theta), s * torch.randn(n, **f)])
    vy = torch.cat([-v * torch.cos(theta), -s * torch.sqrt(-2.0 * torch.log1p(-torch.rand(n, **f)))])
    spc = torch.cat([torch.zeros(n, dtype=torch.int8, device="cuda"), torch.ones(n, dtype=torch.int8, device="cuda")])
    qm = torch.where(spc == 0, E_CHARGE / mass, -E_CHARGE / M_E)
    return x, y, vx, vy, qm, spc


def wall_charge(p, solid, seed):
    """A charge density (C/m^3) like that of a charged-up trench: positive on the floor, negative towards the
    opening, uneven from cell to cell."""
    rng = np.random.default_rng(seed)
    surf = geometry.surface_cells(solid)
    top = p.floor_t + p.trench_d
    depth = (top - np.arange(solid.shape[1]) - 0.5) / p.trench_d
    level = np.where(depth > 0, 1.5 * np.clip(depth, 0, 1) ** 2 - 0.6, 0.0)
    level = np.where(depth > 1, 2.5, level)
    scale = 1.2e4 * (5e-9 / p.dx)
    rho = surf * level[None, :] * scale * rng.uniform(0.7, 1.3, solid.shape)
    rho[:, top:] = 0.0
    return np.where(surf, rho, 0.0)


def prepare(case, seed):
    with torch.no_grad():
        return globals()["prepare_" + case["kind"]](case, seed)


def prepare_step(case, seed):
    p = params_of(case)
    c = ChargingCase(p, circuit=circuit_of(case), max_batches=HISTORY_ROWS)
    n = 2 * p.n_per_batch
    if case["mode"] == "fixed":
        c.load(*particles(p, c.ny, p.n_per_batch, seed))
        c.capture(n)
        return dict(case=c, batch=particles(p, c.ny, p.n_per_batch, seed), n=n)
    tables = (energy_table(), angle_table()) if case["dielectric"] else (None, None)
    inj = inject.DeviceInjector(c, seed=seed, energy_table=tables[0], angle_table=tables[1])
    state = dict(case=c, injector=inj, n=n)
    for _ in range(2):              # a case that has started to charge, as after the first batches of a run
        inj()
        c.step(n)
    c.capture(n)
    return state


def prepare_sweep(case, seed):
    ps, _ = sweep_params(case["cases"], seed=case["shift"])
    b = ChargingBatch(ps, max_batches=HISTORY_ROWS)
    for i, (c, p) in enumerate(zip(b.cases, ps)):
        b.load(i, *particles(p, c.ny, p.n_per_batch, 100 * seed + i))
    b.step()
    b.capture()
    return dict(batch=b)


def prepare_call(case, seed):
    p = params_of(case)
    solid, mask, _, _ = geometry.build_geometry(p)
    vac = ~solid
    ctx = Context(vac, 0, p.dx)
    cond = mask if p.mask_type == "conductor" else np.zeros_like(mask)
    eps = geometry.permittivity(solid, mask, p)
    phi = FieldSolver(ctx, p, eps, cond, False, max_rhs=1).solve((-wall_charge(p, solid, seed) / EPS0).ravel())
    phi = phi.reshape(solid.shape)
    ex, ey = compute_field(phi, vac, p)
    wface = np.where(cond, 1.0, eps / (1.0 + eps))
    parts = [t.cpu().numpy() for t in particles(p, solid.shape[1], p.n_per_batch, seed)]
    return dict(tracer=B200Tracer(vac, precision=case["precision"]), parts=parts, ex=ex, ey=ey, vac=vac, p=p,
                barrier=(phi, wface))


def prepare_setup(case, seed):
    """A case of its own for each seed: another sheet conductance and dielectric."""
    rng = np.random.default_rng(seed)
    p = replace(params_of(case), eps_r=float(rng.uniform(3.6, 4.2)), sigma_s=float(rng.uniform(0.5, 2.0)) * 1e-15,
                field_mode="floating", top_voltage=float(rng.uniform(-5.0, 5.0)))
    return dict(p=p)


def prepare_solve(case, seed):
    p = params_of(case)
    solid, mask, _, _ = geometry.build_geometry(p)
    cond = mask if p.mask_type == "conductor" else np.zeros_like(mask)
    solver = FieldSolver(Context(~solid, 0, p.dx), p, geometry.permittivity(solid, mask, p), cond, False)
    b = np.stack([(-wall_charge(p, solid, 100 * seed + k) / EPS0).ravel() for k in range(case["rhs"])], axis=1)
    return dict(solver=solver, b=b[:, 0].copy() if case["rhs"] == 1 else b, p=p, solid=solid, mask=mask, cond=cond)


def prepare_adjoint(case, seed):
    """A recorded run's histories: hits by table bin and surface slot, and the deposits' response to the charge."""
    p = replace(params_of(case), n_per_batch=1 << 17)
    c = ChargingCase(p, capacity=16, max_batches=HISTORY_ROWS)
    _, e_edges, e_w, a_edges, a_w = adjoint.adjoint_workload()
    rng = np.random.default_rng(seed)
    m, k = c.m, case["modes"]
    rho0 = torch.from_numpy(wall_charge(p, c.solid, seed).ravel()[c.S] * (c.t_sflag.cpu().numpy() & 1 == 0)).cuda()
    h = adjoint.History(c, (e_edges, e_w), (a_edges, a_w), seed, 10, rho0, 0)
    share = rng.dirichlet(np.ones(m))
    for b in range(0, case["batches"], 10):
        nb = min(10, case["batches"] - b)
        by_e = rng.poisson((p.n_per_batch * e_w / e_w.sum())[None, :, None] * share, size=(nb, h.ne, m))
        ions = by_e.sum(axis=1)
        by_a = np.floor((a_w / a_w.sum())[None, :, None] * ions[:, None, :] + rng.random((nb, h.na, m)))
        electrons = rng.poisson(0.98 * ions)
        t = np.concatenate([by_e, by_a, ions[:, None], electrons[:, None]], axis=1).astype(np.int32)
        h.chunks.append(torch.from_numpy(t).pin_memory())
    if k:
        q, _ = np.linalg.qr(rng.standard_normal((m, k)))
        scale = 2e-2 / (c.q_macro / p.dx ** 2) / m
        h.basis = torch.from_numpy(q.copy()).cuda()
        for _ in range(case["batches"]):
            h.resp_i.append(torch.from_numpy(-scale * rng.random((m, k))).cuda())
            h.resp_e.append(torch.from_numpy(scale * rng.random((m, k))).cuda())
            h.resp_index.append(len(h.resp_i) - 1)
    w_e = torch.tensor(e_w, dtype=torch.float64, device="cuda", requires_grad=True)
    w_a = torch.tensor(a_w, dtype=torch.float64, device="cuda", requires_grad=True)
    return dict(hist=h, w_e=w_e, w_a=w_a, rho0=rho0.clone().requires_grad_(True))


# ---- one pass ----------------------------------------------------------------------------

def run(state):
    if "injector" in state:
        state["injector"]()
        state["case"].replay()
        return outputs_of(state["case"], state["n"])
    if "case" in state:
        state["case"].load(*state["batch"])
        state["case"].replay()
        return outputs_of(state["case"], state["n"])
    if "batch" in state:
        state["batch"].replay()
        return [[c.rho_s, c.ex, c.ey, c.hist] for c in state["batch"].cases]
    if "tracer" in state:
        s = state
        cnt_i, cnt_e, escaped, lost = s["tracer"](*s["parts"], s["ex"], s["ey"], s["vac"], s["p"], s["barrier"])
        tallies = np.concatenate([escaped, [lost]]).astype(np.float64)
        return dict(ions=cnt_i.astype(np.float64), electrons=cnt_e.astype(np.float64), tallies=tallies)
    if "solver" in state:
        return state["solver"].solve(state["b"])
    if "hist" in state:
        h = state["hist"]
        for k in ("w_e", "w_a", "rho0"):
            state[k].grad = None
        out = adjoint.objectives(h, state["w_e"], state["w_a"], rho0=state["rho0"])
        (out["phi_bottom"] + out["ratio_i_bottom"].sum()).backward()
        return dict(phi=out["phi_bottom"].detach(), ratio=out["ratio_i_bottom"].detach(), rho=out["rho"].detach(),
                    w_e=state["w_e"].grad, w_a=state["w_a"].grad, rho0=state["rho0"].grad)
    c = ChargingCase(state["p"], max_batches=HISTORY_ROWS)
    return dict(external=c.external, green=c.G, leakage=c.leak_M)


def outputs_of(c, n):
    return dict(rho=c.rho_s, phi=c.phi, ex=c.ex, ey=c.ey, hist=c.hist, monitors=c.qhist, status=c.status[:n])


# ---- what a pass cannot do without -------------------------------------------------------

def grid(case):
    return case["nx"], case["floor"] + case["d"] + case["mask"] + case["vac"]


def surface(case):
    return case["nx"] + 2 * (case["d"] + case["mask"])


def steps_per_particle(case):
    """Mean steps: most particles cross the open vacuum and part of the trench, about a third of a cell a step."""
    opening = case["w"] / case["nx"]
    return (case["vac"] + opening * 0.6 * (case["mask"] + case["d"])) / 0.33


def trace_work(case, n, rf=False):
    steps = n * steps_per_particle(case)
    # a step: bilinear sums 22, weights 8, step length 14, update and wrap 16 (an RF step: two basis fields more)
    return dict(bytes=n * 41.0, flops=steps * (110.0 if rf else 60.0))


def update_work(case):
    nx, ny = grid(case)
    m = surface(case)
    rows = nx * case["vac"] + case["w"] * (case["mask"] + case["d"]) + m
    return dict(bytes=8.0 * m * m + 8.0 * rows * m + 40.0 * nx * ny, flops=2.0 * m * m + 2.0 * rows * m)


def work(case):
    kind = case["kind"]
    if kind == "step":
        a, b = trace_work(case, 2 * case["n"], case["mode"].startswith("rf")), update_work(case)
        return dict(bytes=a["bytes"] + b["bytes"], flops=a["flops"] + b["flops"])
    if kind == "call":
        nx, ny = grid(case)
        a = trace_work(case, 2 * case["n"])
        return dict(bytes=a["bytes"] + 48.0 * nx * ny, flops=a["flops"])
    if kind == "sweep":
        ps, _ = sweep_params(case["cases"], seed=case["shift"])
        total = dict(bytes=0.0, flops=0.0)
        for p in ps:
            c = dict(nx=p.nx, w=p.trench_w, d=p.trench_d, floor=p.floor_t, mask=p.mask_t, vac=p.n_vac)
            for part in (trace_work(c, 2 * p.n_per_batch), update_work(c)):
                total = {k: total[k] + part[k] for k in total}
        return total
    nx, ny = grid(case)
    m = surface(case)
    if kind == "setup":         # the Green's operator written once; multigrid: about 30 cycles of 60 flops a cell
        u = update_work(case)
        return dict(bytes=u["bytes"], flops=m * nx * ny * 1800.0)
    if kind == "solve":
        return dict(bytes=case["rhs"] * nx * ny * 16.0 + 24.0 * nx * ny, flops=case["rhs"] * nx * ny * 1800.0)
    tables = case["batches"] * 98.0 * m * 4
    modes = case["batches"] * case["modes"] * m * 16.0
    return dict(bytes=2 * tables + modes + 8.0 * m * m * 2, flops=case["batches"] * (4.0 * m * m + 4.0 * 98 * m))


def tolerance(case):
    kind = case["kind"]
    if kind in ("setup", "solve"):
        return dict(rel=1e-9, max=1e-7)     # FP64 solves to a relative residual of 1e-13
    if kind == "adjoint":
        return dict(rel=1e-8, max=1e-6)
    if kind == "call" and case["precision"] == "f64":
        # FP64 paths: the counts are the same but for a particle within 1e-13 of an edge
        return dict(rel=1e-6)
    # FP32 paths: about 2 in 10^5 particles land elsewhere under another order of rounding; one particle is a share
    # 1/n of a batch's charge, and later passes carry the difference on
    n = 1 << 17 if kind == "sweep" else 2 * case["n"]
    rel = min(0.03, 4e-4 + 40.0 / n)
    return dict(rel=rel, max=min(1.0, 50 * rel), differ=min(0.01, 1e-4 + 30.0 / n))


# ---- the same result in 64 bits ----------------------------------------------------------

def exact(case, seed):
    """64-bit torch on the same inputs.  None where the result hangs on single particles: of fewer than 2^22
    FP32 paths only a handful land elsewhere than in 64 bits, and which ones is chance."""
    with torch.no_grad():
        if case["kind"] == "step" and case["mode"] == "fixed" and case["n"] >= 1 << 21 and not case["taper"]:
            return exact_step(case, seed)
        if case["kind"] == "call" and case["precision"] == "f64" and not (case["taper"] or case["mask_taper"]):
            return exact_call(case, seed)
        if case["kind"] == "setup":
            return exact_setup(case, seed)
        if case["kind"] == "solve":
            return exact_solve(case, seed)
    if case["kind"] == "adjoint":
        return exact_adjoint(case, seed)
    return None


def dense_operator(eps, cond, p):
    """The 5-point finite-volume operator div(eps grad) of a periodic trench as a dense 64-bit matrix."""
    nx, ny = eps.shape
    e, c = torch.from_numpy(eps).cuda(), torch.from_numpy(cond).cuda()

    def face(a, b, ca, cb):
        h = torch.where(ca, 2.0 * b, torch.where(cb, 2.0 * a, 2.0 * a * b / (a + b)))
        return torch.where(ca & cb, torch.zeros_like(h), h) / p.dx ** 2

    east = face(e, torch.roll(e, -1, 0), c, torch.roll(c, -1, 0))
    north = face(e[:, :-1], e[:, 1:], c[:, :-1], c[:, 1:])
    diag = -(east + torch.roll(east, 1, 0))
    diag[:, :-1] -= north
    diag[:, 1:] -= north
    diag[:, 0] -= 2.0 * e[:, 0] / p.dx ** 2
    diag[:, -1] -= 2.0 * e[:, -1] / p.dx ** 2
    idx = torch.arange(nx * ny, device="cuda").reshape(nx, ny)
    A = torch.zeros((nx * ny, nx * ny), dtype=torch.float64, device="cuda")
    A[idx.ravel(), idx.ravel()] = diag.ravel()
    right = torch.roll(idx, -1, 0)
    A[idx.ravel(), right.ravel()] += east.ravel()
    A[right.ravel(), idx.ravel()] += east.ravel()
    A[idx[:, :-1].ravel(), idx[:, 1:].ravel()] = north.ravel()
    A[idx[:, 1:].ravel(), idx[:, :-1].ravel()] = north.ravel()
    return A


class DenseSolver:
    """A phi = b by LU: a floating conductor is one unknown, a driven one is held at zero."""

    def __init__(self, eps, cond, p, driven):
        self.A = dense_operator(eps, cond, p)
        flat = torch.from_numpy(cond.ravel()).cuda()
        self.free = torch.nonzero(~flat).ravel()
        self.held = torch.nonzero(flat).ravel()
        self.one = bool(len(self.held)) and not driven
        M = self.A[self.free][:, self.free]
        if self.one:
            edge = self.A[self.free][:, self.held].sum(1)
            corner = self.A[self.held][:, self.held].sum()
            M = torch.cat([torch.cat([M, edge[:, None]], 1), torch.cat([edge, corner[None]])[None, :]], 0)
        self.M = M
        self.lu, self.piv = torch.linalg.lu_factor(M)

    def __call__(self, b):
        """b (n, k) -> phi (n, k), with one step of refinement."""
        r = b[self.free]
        if self.one:
            r = torch.cat([r, b[self.held].sum(0, keepdim=True)])
        x = torch.linalg.lu_solve(self.lu, self.piv, r)
        x = x + torch.linalg.lu_solve(self.lu, self.piv, r - self.M @ x)
        phi = torch.zeros_like(b)
        phi[self.free] = x[:len(self.free)]
        if self.one:
            phi[self.held] = x[-1]
        return phi


def leak_operator(p, solid, P, S):
    """inv(I - dt G_leak P) of the sheet conductance between neighbouring surface cells (S, flat)."""
    nx, ny = solid.shape
    slot = -np.ones(nx * ny, dtype=np.int64)
    slot[S] = np.arange(len(S))
    slot = slot.reshape(nx, ny)
    g = torch.zeros((len(S), len(S)), dtype=torch.float64, device="cuda")
    c = torch.tensor(p.sigma_s / p.dx, dtype=torch.float64, device="cuda")
    for a, b in ((slot, np.roll(slot, -1, 0)), (slot[:, :-1], slot[:, 1:])):
        ok = (a >= 0) & (b >= 0)
        i, j = torch.from_numpy(a[ok]).cuda(), torch.from_numpy(b[ok]).cuda()
        for r, s, v in ((i, j, c), (j, i, c), (i, i, -c), (j, j, -c)):
            g.index_put_((r, s), v.expand(len(r)), accumulate=True)
    eye = torch.eye(len(S), dtype=torch.float64, device="cuda")
    return torch.linalg.inv(eye - p.dt_batch * (g @ P)), g


def materials(p):
    solid, mask, _, _ = geometry.build_geometry(p)
    cond = mask if p.mask_type == "conductor" else np.zeros_like(mask)
    eps = np.where(solid, p.eps_r, 1.0)
    if p.mask_type == "dielectric":
        eps = np.where(mask, p.mask_eps_r, eps)
    return solid, mask, cond, eps


def exact_solve(case, seed):
    p = params_of(case)
    solid, _, cond, eps = materials(p)
    b = np.stack([(-wall_charge(p, solid, 100 * seed + k) / EPS0).ravel() for k in range(case["rhs"])], axis=1)
    x = DenseSolver(eps, cond, p, False)(torch.from_numpy(b).cuda()).cpu().numpy()
    return x[:, 0].copy() if case["rhs"] == 1 else x


def boundary(p, eps):
    """Right-hand side of the substrate and top potentials."""
    rhs = np.zeros_like(eps)
    rhs[:, 0] -= 2.0 * eps[:, 0] / p.dx ** 2 * p.substrate_voltage
    rhs[:, -1] -= 2.0 * eps[:, -1] / p.dx ** 2 * p.top_voltage
    return torch.from_numpy(rhs.ravel()).cuda()


def green_of(solve, n, S, driven, cond):
    """Potential everywhere per unit charge density on each surface cell, (n, m)."""
    b = torch.zeros((n, len(S)), dtype=torch.float64, device="cuda")
    b[torch.from_numpy(S).cuda(), torch.arange(len(S), device="cuda")] = -1.0 / EPS0
    return solve(b)


def surface_set(solid):
    vac = ~solid
    near = vac | np.roll(vac, 1, 0) | np.roll(vac, -1, 0)
    wide = near.copy()
    wide[:, 1:] |= near[:, :-1]
    wide[:, :-1] |= near[:, 1:]
    return solid & wide


def exact_setup(case, seed):
    p = prepare_setup(case, seed)["p"]
    solid, mask, cond, eps = materials(p)
    solve = DenseSolver(eps, cond, p, False)
    S = np.flatnonzero(surface_set(solid).ravel())
    G = green_of(solve, solid.size, S, False, cond)
    rows = np.flatnonzero((~solid | surface_set(solid)).ravel())
    probes = [ix * solid.shape[1] + iy for ix, iy in geometry.probe_cells(solid, p, bool(cond.any())).values()]
    rows = np.union1d(rows, probes)
    M, _ = leak_operator(p, solid, G[torch.from_numpy(S).cuda()] / p.dx ** 2, S)
    external = solve(boundary(p, eps)[:, None])[:, 0].reshape(solid.shape)
    return dict(external=external.cpu().numpy(), green=G[torch.from_numpy(rows).cuda()], leakage=M)


def wall_entry(x0, y0, sx, sy, vac, dx, nx, ny):
    """The first solid face that a move crosses: its cell, the vacuum cell before it, whether it is an x face."""
    ix0, iy0 = (x0 / dx).long().clamp(max=nx - 1), (y0 / dx).long().clamp(0, ny - 1)
    dix = torch.floor((x0 + sx) / dx).long() - ix0
    diy = torch.floor((y0 + sy) / dx).long().clamp(0, ny - 1) - iy0
    inf = torch.full_like(x0, math.inf)
    fx = torch.where(dix != 0, ((ix0 + (dix > 0)) * dx - x0) / sx, inf)
    fy = torch.where(diy != 0, ((iy0 + (diy > 0)) * dx - y0) / sy, inf)
    x_first = fx < fy
    ax = torch.where(x_first, (ix0 + dix) % nx, ix0)
    ay = torch.where(x_first, iy0, iy0 + diy)
    last = (dix != 0) & (diy != 0) & (vac[ax * ny + ay] > 0)
    cx, cy = torch.where(last, (ix0 + dix) % nx, ax), torch.where(last, iy0 + diy, ay)
    vx, vy = torch.where(last, ax, ix0), torch.where(last, ay, iy0)
    return cx * ny + cy, vx * ny + vy, torch.where(last, ~x_first, x_first)


def trace64(parts, ex, ey, solid, p, phi, wface):
    """Straight-walled barrier tracing in 64 bits, all particles a step at a time: hits per species and cell,
    escaped per species, lost."""
    x, y, vx, vy, qm, spc = (t.clone() for t in parts)
    spc = spc.long()
    nx, ny = solid.shape
    dx, lx, ly = p.dx, nx * p.dx, ny * p.dx
    vac = torch.from_numpy((~solid).ravel().astype(np.float64)).cuda()
    exv, eyv = ex.ravel() * vac, ey.ravel() * vac
    phi, wface = phi.ravel(), wface.ravel()
    hits = torch.zeros(2 * nx * ny, dtype=torch.float64, device="cuda")
    escaped = torch.zeros(2, dtype=torch.float64, device="cuda")
    for _ in range(p.max_steps):
        if not len(x):
            break
        fx, fy = x / dx - 0.5, y / dx - 0.5
        i0, j0 = torch.floor(fx), torch.floor(fy)
        tx, ty = fx - i0, fy - j0
        i0, j0 = i0.long(), j0.long()
        i1, i0 = (i0 + 1) % nx, i0 % nx
        j1, j0 = (j0 + 1).clamp(0, ny - 1), j0.clamp(0, ny - 1)
        corners = ((i0 * ny + j0, (1 - tx) * (1 - ty)), (i1 * ny + j0, tx * (1 - ty)),
                   (i0 * ny + j1, (1 - tx) * ty), (i1 * ny + j1, tx * ty))
        sx = sum(w * exv[c] for c, w in corners)
        sy = sum(w * eyv[c] for c, w in corners)
        sw = sum(w * vac[c] for c, w in corners).clamp(min=1e-12)
        ax, ay = qm * (sx / sw), qm * (sy / sw)
        dt = p.cfl * dx / (torch.hypot(vx, vy) + torch.sqrt(2.0 * dx * torch.hypot(ax, ay)) + 1.0)
        vxn, vyn = vx + ax * dt, vy + ay * dt
        mx, my = 0.5 * (vx + vxn) * dt, 0.5 * (vy + vyn) * dt
        xn, yn = torch.remainder(x + mx, lx), y + my
        out = yn >= ly
        cell = (xn / dx).long().clamp(max=nx - 1) * ny + (yn / dx).long().clamp(0, ny - 1)
        hit = ~out & (vac[cell] == 0)
        h = torch.nonzero(hit).ravel()
        if len(h):
            cc, vv, face_x = wall_entry(x[h], y[h], mx[h], my[h], vac, dx, nx, ny)
            vn = torch.where(face_x, vxn[h], vyn[h])
            back = 0.5 * (vn * vn) < qm[h] * (wface[cc] * (phi[cc] - phi[vv]))
            b, fb = h[back], face_x[back]
            vxn[b] = torch.where(fb, -vxn[b], vxn[b])
            vyn[b] = torch.where(fb, vyn[b], -vyn[b])
            xn[b], yn[b] = x[b], y[b]
            hit[b] = False
            stay = ~back
            hits.index_add_(0, spc[h[stay]] * (nx * ny) + cc[stay], torch.ones(int(stay.sum()), dtype=torch.float64,
                                                                               device="cuda"))
        escaped.index_add_(0, spc[out], torch.ones(int(out.sum()), dtype=torch.float64, device="cuda"))
        live = ~(hit | out)
        x, y, vx, vy, qm, spc = xn[live], yn[live], vxn[live], vyn[live], qm[live], spc[live]
    return hits.reshape(2, nx, ny), escaped, len(x)


def exact_call(case, seed):
    s = prepare_call(case, seed)
    f = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    hits, escaped, lost = trace64([f(a) for a in s["parts"]], f(s["ex"]), f(s["ey"]), ~s["vac"], s["p"],
                                  f(s["barrier"][0]), f(s["barrier"][1]))
    return dict(ions=hits[0].cpu().numpy(), electrons=hits[1].cpu().numpy(),
                tallies=np.array([*escaped.cpu().numpy(), lost], dtype=np.float64))


def gradient(phi, vac, p):
    """E = -grad phi over vacuum neighbours."""
    ghost_top, ghost_bottom = 2 * p.top_voltage - phi[:, -1:], 2 * p.substrate_voltage - phi[:, :1]
    no = torch.zeros_like(vac[:, :1])

    def one(m, pl, vm, vp):
        g = torch.where(vm & vp, (pl - m) / (2 * p.dx), torch.zeros_like(phi))
        g = torch.where(vp & ~vm, (pl - phi) / p.dx, g)
        return -torch.where(vm & ~vp, (phi - m) / p.dx, g)

    ex = one(torch.roll(phi, 1, 0), torch.roll(phi, -1, 0), torch.roll(vac, 1, 0), torch.roll(vac, -1, 0))
    ey = one(torch.cat([ghost_bottom, phi[:, :-1]], 1), torch.cat([phi[:, 1:], ghost_top], 1),
             torch.cat([no, vac[:, :-1]], 1), torch.cat([vac[:, 1:], ~no], 1))
    return ex, ey


def exact_step(case, seed):
    """The first batch of a run under fixed voltages: trace, deposit, leakage, potential, field."""
    p = params_of(case)
    solid, mask, cond, eps = materials(p)
    nx, ny = solid.shape
    solve = DenseSolver(eps, cond, p, True)
    held = torch.from_numpy(cond.ravel()).cuda()
    phi_c = held.double() * p.mask_voltage
    external = solve((boundary(p, eps) - solve.A @ phi_c)[:, None])[:, 0] + phi_c
    S = np.flatnonzero(surface_set(solid).ravel())
    ts = torch.from_numpy(S).cuda()
    b = torch.zeros((nx * ny, len(S)), dtype=torch.float64, device="cuda")
    b[ts, torch.arange(len(S), device="cuda")] = -1.0 / EPS0
    G = solve(torch.where(held[:, None], torch.zeros_like(b), b))
    M, g = leak_operator(p, solid, G[ts] / p.dx ** 2, S)
    vac = torch.from_numpy(~solid).cuda()
    ex, ey = gradient(external.reshape(nx, ny), vac, p)
    wface = torch.from_numpy(np.where(cond, 1.0, eps / (1.0 + eps))).cuda()
    parts = particles(p, ny, p.n_per_batch, seed)
    hits, _, _ = trace64(parts, ex, ey, solid, p, external, wface)
    hits = hits.reshape(2, -1)
    q = E_CHARGE * (p.flux * (nx * p.dx) * p.dt_batch / p.n_per_batch)
    rho = torch.where(held[ts], torch.zeros(len(S), dtype=torch.float64, device="cuda"),
                      (hits[0] - hits[1])[ts] * q / p.dx ** 2)
    rho = (M @ (rho * p.dx ** 2 + p.dt_batch * (g @ external[ts]))) / p.dx ** 2
    rho = torch.where(held[ts], torch.zeros_like(rho), rho)
    full = external + G @ rho
    rows = torch.from_numpy((~solid | surface_set(solid)).ravel()).cuda()
    for ix, iy in geometry.probe_cells(solid, p, bool(cond.any())).values():
        rows[ix * ny + iy] = True
    phi = torch.where(rows, full, external)
    ex, ey = gradient(phi.reshape(nx, ny), vac, p)
    return dict(rho=rho, phi=phi, ex=ex.ravel(), ey=ey.ravel(), hist=None, monitors=None, status=None)


def exact_adjoint(case, seed):
    """The recurrence over the recorded histories in 64-bit torch, differentiated by torch.autograd."""
    s = prepare_adjoint(case, seed)
    h = s["hist"]
    c = h.case
    p, m, dev = c.p, c.m, "cuda"
    flag = c.t_sflag.long()
    cond, bottom = (flag & 1) != 0, (flag & 4) != 0
    leak_M, leak_h, g_s = c.leak_M, c.leak_h, c.g_s
    w_e, w_a, rho0 = s["w_e"], s["w_a"], s["rho0"]
    T = torch.cat(h.chunks).to(dev).double()
    r_e = w_e / w_e.sum() / (w_e.detach() / w_e.detach().sum())
    r_a = w_a / w_a.sum() / (w_a.detach() / w_a.detach().sum())
    dx2, q = p.dx ** 2, c.q_macro
    rho, ratio = rho0, []
    for b in range(len(T)):
        ci = T[b, h.ne + h.na] + (r_e - 1) @ T[b, :h.ne] + (r_a - 1) @ T[b, h.ne:h.ne + h.na]
        ce = T[b, h.ne + h.na + 1]
        if h.has_feedback:
            shift = h.basis.T @ (rho - rho.detach())
            ci = ci + h.resp_i[b] @ shift
            ce = ce + h.resp_e[b] @ shift
        r = rho + torch.where(cond, torch.zeros_like(ci), (ci - ce) * q / dx2)
        if leak_M is not None:
            r = leak_M @ (r * dx2 + (leak_h if leak_h is not None else 0.0)) / dx2
        if c.floating:
            drift = dx2 * (g_s * (r - rho)).sum()
            x_i, x_e = q * ci[cond].sum() / c.C_cond + drift, q * ce[cond].sum() / c.C_cond
            k = x_i / p.electron_temp_eV
            frac = -torch.expm1(-k) / k
            dv = -p.electron_temp_eV * torch.logaddexp(-k, torch.log(x_e / p.electron_temp_eV * frac))
            unit = torch.zeros(m, dtype=torch.float64, device=dev)
            unit[c.c_slot] = 1.0
            r = r + unit * (c.C_cond * (dv - drift) / dx2)
        rho = r
        ratio.append(ci[bottom].sum() / (p.n_per_batch * ((c.b1 - c.b0) / c.nx)))
    ix, iy = c.probes["bottom center"]
    cell = ix * c.ny + iy
    solid, mask, cond_cells, eps = materials(p)
    with torch.no_grad():
        solve = DenseSolver(eps, cond_cells, p, False)
        unit = torch.zeros((solid.size, 1), dtype=torch.float64, device=dev)
        unit[cell] = 1.0
        row = -solve(unit)[:, 0][c.t_surf.long()] / EPS0
    ratio = torch.stack(ratio)
    phi = c.t_ext[cell] + row @ rho
    (phi + ratio.sum()).backward()
    return dict(phi=phi.detach(), ratio=ratio.detach(), rho=rho.detach(), w_e=w_e.grad, w_a=w_a.grad,
                rho0=rho0.grad)
