"""The coarsest algebraic inverse at sizes around its 32-pivot blocks and 128 x 64 tiles: with all
vertices of the mesh inverted densely the V-cycle's coarse correction is exact, so the iteration
count stays that of the smallest mesh; a wrong block would show as many more."""
import numpy as np
import pytest

import sipg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("singular", [False, True])
@pytest.mark.parametrize("n", [3, 4, 5, 7, 10, 11, 15, 22, 27])  # (n + 1)^2 = 16 ... 784 unknowns
def test_exact_coarse_correction(n, singular):
    mesh = sipg.Mesh.box(2, n, jitter=0.1, seed=2)
    op = sipg.Operator(mesh, 2, 1)
    op.set_bc_types(np.full((1, mesh.Kb), sipg.BC_NEUMANN if singular else sipg.BC_DIRICHLET, np.int32))
    o = sipg.default_opts(sipg.SOLVER_PMULTIGRID)
    o.n_levels, o.orders[0], o.orders[1] = 2, 2, 1
    o.rel_tol, o.abs_tol, o.nullspace = 1e-10, 0.0, int(singular)
    b = np.random.default_rng(n).uniform(-1, 1, op.shape())
    b -= b.mean()
    x, info = sipg.Solver(op, sipg.SOLVER_PMULTIGRID, o).solve_host(b)
    assert info.status == 0 and info.true_rel_res < 1e-9
    assert info.iters <= 20
