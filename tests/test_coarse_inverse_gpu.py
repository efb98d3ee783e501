"""The coarsest algebraic inverse at sizes around its 32-pivot blocks and 128 x 64 tiles: the
inversion by itself against the host's, and in a solve. There all vertices of the mesh are inverted
densely, so that the V-cycle's coarse correction is exact and the solve takes at most 20 iterations
on every mesh; damage that slows it more than that shows, smaller damage only in the inversion's
own test."""
import ctypes as C

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


def spd(n, rng):
    """Symmetric with eigenvalues in [1, 10]."""
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * rng.uniform(1.0, 10.0, n)) @ q.T
    return 0.5 * (a + a.T)


@pytest.mark.parametrize("project", [False, True])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 191, 193, 257, 400])
def test_dense_inverse(n, project):
    """The inversion itself, at remainders of the 32-pivot blocks and 128 x 64 tiles and at odd and
    even numbers of steps (an odd one is copied back): A X = I up to the elimination's rounding, at
    most n eps per entry times the condition number squared (100)."""
    rng = np.random.default_rng(n)
    a = spd(n, rng)
    # dense_inverse_device(double* a, int n, bool project_constants, double* work, cudaStream_t)
    inverse = sipg.lib()["_ZN4sipg20dense_inverse_deviceEPdibS0_P11CUstream_st"]
    inverse.restype = None
    da = sipg.DeviceVector(a)
    work = sipg.DeviceVector(np.full(n * n + 2 * n + 2048, np.nan))
    inverse(C.c_void_p(da.ptr), C.c_int(n), C.c_bool(project), C.c_void_p(work.ptr), C.c_void_p(0))
    got = da.get().reshape(n, n)
    want = np.linalg.inv(a)
    if project:
        q = np.eye(n) - 1.0 / n
        want = q @ want @ q
    bound = n * np.finfo(np.float64).eps * 100.0
    assert np.abs(got - want).max() < bound
    if not project:
        assert np.abs(a @ got - np.eye(n)).max() < 10.0 * bound
