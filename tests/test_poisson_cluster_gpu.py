"""The one-launch Poisson solve (one cluster to a right-hand side) at the edges of its range: the grid
sizes where the dispatch or the shared-memory layout changes, odd and narrow grids.
"""
from dataclasses import replace

import numpy as np
import pytest

from trench_b200 import geometry
from trench_b200.params import Params

pytestmark = pytest.mark.gpu


# one and two levels (the launch per pass); three levels; odd widths (four colours); more CTAs than
# columns; 60 x 250 (two right-hand sides fit a cluster) and 80 x 294 (one does); the
# largest blocks (7 cells a thread) and the first grids beyond them
@pytest.mark.parametrize("shape", [(5, 9), (12, 16), (16, 17), (21, 33), (33, 40), (60, 100), (61, 250), (60, 250),
                                   (80, 294), (79, 293), (81, 294), (80, 299), (120, 273), (2, 40), (4, 90)])
@pytest.mark.parametrize("rhs", [1, 5, 19])
def test_solutions_satisfy_the_operator(cuda_device, shape, rhs):
    """|b - L x| <= rtol |b| in FP64 (or the residual's own rounding floor), for right-hand sides of
    very different smoothness, which converge after different numbers of refinements."""
    import torch
    from trench_b200.fields import FieldSolver, apply_matrix
    from trench_b200.tracer import Context
    nx, ny = shape
    rng = np.random.default_rng(nx * 1000 + ny)
    p = replace(Params(), nx=nx, floor_t=1, trench_d=1)
    eps = np.where(rng.random(shape) < 0.4, 3.9, 1.0)
    cond = np.zeros(shape, bool)
    if nx > 8:
        cond[2:5, ny // 3:ny // 2] = True
    solver = FieldSolver(Context(np.ones(shape, bool), cuda_device, p.dx), p, eps, cond, True, max_rhs=20)
    b = np.zeros((rhs, nx * ny))
    b[0] = rng.normal(0, 1, nx * ny)
    for k in range(1, rhs):
        b[k, rng.integers(nx * ny)] = 10.0 ** (k % 7)          # point charges of different size
    b[:, cond.ravel()] = 0.0
    x = solver.solve_rows(torch.from_numpy(b).cuda() / solver.dx2).cpu().numpy()
    for k in range(rhs):
        phi = x[k].reshape(shape)
        r = (apply_matrix(solver.diag, solver.ce, solver.cn, phi) * solver.dx2).ravel() - b[k]
        r[cond.ravel()] = 0.0
        # the magnitude of the terms bounds the rounding of the residual computed here
        size = (apply_matrix(np.abs(solver.diag), solver.ce, solver.cn, np.abs(phi)) * solver.dx2).ravel()
        bound = max(2 * solver.rtol * np.linalg.norm(b[k]),
                    64 * np.finfo(float).eps * (np.linalg.norm(size) + np.linalg.norm(b[k])))
        assert np.linalg.norm(r) <= bound
        assert np.all(phi[cond] == 0.0)


def test_right_hand_sides_do_not_depend_on_their_block(cuda_device):
    """One right-hand side alone gives the bits it gives in a block."""
    import torch
    from trench_b200.fields import FieldSolver
    from trench_b200.tracer import Context
    p = replace(Params(), nx=40, trench_w=14, trench_d=50)
    solid, mask, _, _ = geometry.build_geometry(p)
    eps = geometry.permittivity(solid, mask, p)
    solver = FieldSolver(Context(~solid, cuda_device, p.dx), p, eps, np.zeros_like(mask), False, max_rhs=300)
    b = torch.randn((300, solid.size), dtype=torch.float64, device="cuda")
    block = solver.solve_rows(b)
    for k in (0, 149, 299):
        assert torch.equal(solver.solve_rows(b[k:k + 1])[0], block[k])
