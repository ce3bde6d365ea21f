"""What tb_poisson_solve promises beyond its tolerance, at the C entry: the smoother's full division, and
a guess within the tolerance left as it is; and the hierarchy built once where a case's set-up has
no work vectors to give back."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def four_squares(r):
    a = math.isqrt(r)
    while True:
        b = math.isqrt(r - a * a)
        while b >= 0 and r - a * a - b * b < 1 << 20:
            rest = r - a * a - b * b
            for c in range(math.isqrt(rest) + 1):
                d = math.isqrt(rest - c * c)
                if c * c + d * d == rest:
                    return a, b, c, d
            b -= 1
        a -= 1


def setup(shape, diag, ke, kn, max_rhs):
    from trench_b200 import _capi
    from trench_b200.tracer import Context
    ctx = Context(np.ones(shape, bool), 0, 1.0)
    ptr = lambda a: np.ascontiguousarray(a).ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    arrays = [np.ascontiguousarray(a, dtype=np.float64) for a in (diag, ke, kn)] + [np.zeros(shape, np.uint8)]
    ctx.check(_capi.lib().tb_poisson_setup(ctx.handle, *(ptr(a) for a in arrays), max_rhs))
    return ctx


def solve(ctx, b, x, rtol=1e-13, max_outer=40, inner=12):
    """(return code, refinement steps, residual); x is the guess and the solution, on the device."""
    from trench_b200 import _capi
    from trench_b200.tracer import _ptr
    iters, resid = ctypes.c_int(), ctypes.c_double()
    rc = _capi.lib().tb_poisson_solve(ctx.handle, len(b), _ptr(b), _ptr(x), rtol, max_outer, inner, ctypes.byref(iters),
                                      ctypes.byref(resid), None)
    return rc, iters.value, resid.value


# whole solve in one launch (one and two sides to a cluster); all levels in one CTA; odd widths
@pytest.mark.parametrize("shape", [(60, 100), (21, 33), (4, 90)])
@pytest.mark.parametrize("rhs", [1, 20])
def test_the_smoother_divides_in_full(cuda_device, shape, rhs):
    """Without couplings one smoothing step is b / d.  With b = +-d, |b| a power of two and so every
    scaled number exact, one PCG iteration gives +-1 to the last bit, if and only if the FP32
    quotients are correctly rounded."""
    import torch
    rng = np.random.default_rng(shape[0])
    n = shape[0] * shape[1]
    d = 2.0 * rng.integers(1, 2048, n) + 1
    want = rng.choice([-1.0, 1.0], n)
    d[-4:] = 1.0
    s = int((d[:-4] ** 2).sum())
    m = 1
    while 4 ** m < s:
        m += 1
    want[-4:] = four_squares(4 ** m - s)
    b = d * want
    ctx = setup(shape, d.reshape(shape), np.zeros(shape), np.zeros(shape), 20)
    B = torch.from_numpy(np.tile(b, (rhs, 1))).cuda()
    X = torch.zeros_like(B)
    rc, iters, resid = solve(ctx, B, X, max_outer=1, inner=1)
    assert (rc, iters, resid) == (0, 1, 0.0)
    np.testing.assert_array_equal(X.cpu().numpy(), np.tile(want, (rhs, 1)))
    ctx.close()


# one launch (one and two sides to a cluster), and a launch per pass
@pytest.mark.parametrize("shape", [(60, 100), (60, 600)])
@pytest.mark.parametrize("rhs", [1, 20])
def test_a_guess_within_the_tolerance_is_kept(cuda_device, shape, rhs):
    import torch
    rng = np.random.default_rng(8)
    ke = np.ones(shape)
    kn = np.ones(shape)
    kn[:, -1] = 0.0
    diag = 4.0 + np.zeros(shape)
    diag[:, 0] += 1.0
    diag[:, -1] += 1.0
    ctx = setup(shape, diag, ke, kn, 20)
    B = torch.from_numpy(rng.normal(0, 1, (rhs, shape[0] * shape[1]))).cuda()
    X = torch.zeros_like(B)
    rc, iters, resid = solve(ctx, B, X, rtol=1e-6)
    assert rc == 0 and iters >= 1 and resid <= 1e-6
    guess = X.clone()
    # twice the residual as the tolerance: within it, though not within a tenth of it
    rc, iters, again = solve(ctx, B, X, rtol=2 * resid)
    assert (rc, iters) == (0, 0) and torch.equal(X, guess)
    rc, iters, again = solve(ctx, B, X, rtol=resid / 2)
    assert rc == 0 and iters >= 1 and again <= resid / 2
    ctx.close()


@pytest.mark.parametrize("depth,times", [(160, 1), (500, 2)])
def test_set_up_builds_the_hierarchy_once(cuda_device, monkeypatch, depth, times):
    """60 x 250 cells: one launch, no work vectors.  60 x 590 cells with 1100 surface cells: 1.7 GB of
    them, released by a second, narrow set-up."""
    from dataclasses import replace
    from trench_b200.fields import FieldSolver
    from trench_b200.params import Params
    from trench_b200.step import ChargingCase
    built = []
    setup_once = FieldSolver._setup
    monkeypatch.setattr(FieldSolver, "_setup", lambda self, k: (built.append(k), setup_once(self, k)))
    p = replace(Params(), nx=60, trench_w=20, trench_d=depth, floor_t=10, mask_t=20, n_vac=60)
    c = ChargingCase(p, capacity=16, max_batches=4)
    assert len(built) == times
    assert built[0] >= c.m
    if times == 1:
        assert c.solver.side_bytes * c.solver.max_rhs < 1 << 20
    else:
        assert c.solver.side_bytes > 40 * c.n and c.solver.max_rhs == 64


def test_many_sides_of_a_small_grid(cuda_device):
    """300 sides of 840 cells go by launches, 100 by one launch: the same solutions."""
    import torch
    shape, rhs = (12, 70), 300
    rng = np.random.default_rng(3)
    kn = rng.uniform(0.5, 4.0, shape)
    kn[:, -1] = 0.0
    ke = rng.uniform(0.5, 4.0, shape)
    diag = ke + np.roll(ke, 1, axis=0) + kn + np.pad(kn, ((0, 0), (1, 0)))[:, :-1]
    diag[:, [0, -1]] += 2.0
    ctx = setup(shape, diag, ke, kn, rhs)
    B = torch.from_numpy(rng.normal(0, 1, (rhs, 840))).cuda()
    X, Y = torch.zeros_like(B), torch.zeros_like(B)
    rc, iters, resid = solve(ctx, B, X)
    assert rc == 0 and resid <= 1e-13
    for s in (0, 100, 200):
        rc, iters, resid = solve(ctx, B[s:s + 100].contiguous(), Y[s:s + 100])
        assert rc == 0 and resid <= 1e-13
    # |x - y| <= |L^-1| (|r_x| + |r_y|); the smallest eigenvalue of this operator is above 0.002
    assert float((X - Y).norm(dim=1).max()) <= 2e-13 / 0.002 * float(B.norm(dim=1).max())
    ctx.close()
