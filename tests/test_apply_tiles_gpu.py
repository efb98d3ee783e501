"""Edges of the tensor-core apply's warp tiles (8 elements FP64, 16 FP32): meshes below one
tile, exactly some tiles and with a remainder, a pinned DOF in the last tile, and the
in-place apply (y over x), at every order in 2D and 3D."""
import numpy as np
import pytest

import oracle_py as O
import sipg
from helpers import TOL_FP64, TOL_TF32, DevArray, make_op, random_case, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("dim,n", [(2, 1), (2, 4), (2, 5), (3, 1), (3, 2), (3, 3)])
def test_tile_edges_pin_and_in_place(dim, n, order):
    mesh, t, e, om, x, f, m, bct = random_case(dim, n, order, 1, seed=7 * order + dim)
    op = make_op(mesh, order, 1, f, bct=bct)
    K, Np = mesh.K, x.shape[2]
    op.set_pin(K - 1, Np - 1)
    xs = x.copy()
    xs[0, K - 1, Np - 1] = 0.0
    ref = O.mult(om, xs, bct, f)
    ref[0, K - 1, Np - 1] = O.diag(om, 1, bct, f)[0, K - 1, Np - 1] * x[0, K - 1, Np - 1]
    for prec, dtype, tol in ((sipg.FP64, np.float64, TOL_FP64), (sipg.FP32, np.float32, TOL_TF32)):
        xd, yd = DevArray(x.astype(dtype)), DevArray(np.full(x.shape, 7.0, dtype))
        op.apply_device(prec, xd.p, yd.p)
        y = yd.get()
        assert rel_err(y.astype(np.float64), ref) < tol
        op.apply_device(prec, xd.p, xd.p)  # every tile reads its own rows before it writes them
        assert np.array_equal(xd.get(), y)


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("dim,n", [(2, 5), (2, 7), (3, 1), (3, 3)])
def test_vector_operator_with_slip_faces(dim, n, order):
    """All components in one launch, or one after the other where a component's rows do not
    start on 16 bytes (2D p = 1, n = 5 and 7 in FP32: 150 and 294 values)."""
    mesh, t, e, om, x, f, m, bct = random_case(dim, n, order, dim, seed=3 * order + dim, slip=True, mm=True)
    op = make_op(mesh, order, dim, f, m, bct=bct)
    ref = O.mult(om, x, bct, f, m)
    for prec, dtype, tol in ((sipg.FP64, np.float64, TOL_FP64), (sipg.FP32, np.float32, TOL_TF32)):
        xd, yd = DevArray(x.astype(dtype)), DevArray(np.full(x.shape, 7.0, dtype))
        op.apply_device(prec, xd.p, yd.p)
        assert rel_err(yd.get().astype(np.float64), ref) < tol


@pytest.mark.parametrize("kernel", [2, 3])
@pytest.mark.parametrize("prec,dtype,tol", [(sipg.FP64, np.float64, TOL_FP64), (sipg.FP32, np.float32, TOL_TF32)],
                         ids=["fp64", "fp32"])
@pytest.mark.parametrize("dim,n,order", [(2, 4, 2), (3, 2, 3), (3, 3, 4)])
def test_vector_operator_first_apply_with_a_selected_kernel(dim, n, order, kernel, prec, dtype, tol):
    """The first apply of a vector operator allocates the trace scratch under every tensor-core
    kernel selection, the component-by-component one (3) included."""
    mesh, t, e, om, x, f, m, bct = random_case(dim, n, order, dim, seed=order + dim, slip=True, mm=True)
    op = make_op(mesh, order, dim, f, m, bct=bct)
    op.set_kernel(kernel)
    xd, yd = DevArray(x.astype(dtype)), DevArray(np.full(x.shape, 7.0, dtype))
    op.apply_device(prec, xd.p, yd.p)
    assert rel_err(yd.get().astype(np.float64), O.mult(om, x, bct, f, m)) < tol


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("dim,n", [(2, 4), (2, 5), (3, 1), (3, 3)])
def test_fp32_slip_terms_are_not_rounded_to_tf32(dim, n, order):
    """The slip faces' terms of the FP32 vector operator, isolated as the difference to the same
    operator with natural faces there, agree with the FP64 ones to FP32 accuracy, whether the
    components' rows start on 16 bytes or not: an FP32 sum of up to 115 products (node and face-node
    sums one after the other) is off by at most 115 * 2^-24 = 7e-6 of the terms' size, which the
    gradient's cancellation can raise a few times; operands rounded to TF32 (10 bits) give 2e-4 and
    more."""
    mesh, t, e, om, x, f, m, bct = random_case(dim, n, order, dim, seed=11 * order + dim, slip=True, mm=True)
    natural = np.where(bct == sipg.BC_SLIP, sipg.BC_NEUMANN, bct).astype(np.int32)
    terms = {}
    for prec, dtype in ((sipg.FP64, np.float64), (sipg.FP32, np.float32)):
        y = []
        for types in (bct, natural):
            op = make_op(mesh, order, dim, f, m, bct=types)
            xd, yd = DevArray(x.astype(np.float32).astype(dtype)), DevArray(np.zeros(x.shape, dtype))
            op.apply_device(prec, xd.p, yd.p)
            y.append(yd.get().astype(np.float64))
        terms[prec] = y[0] - y[1]
        size = np.abs(y[0]).max()
    assert np.abs(terms[sipg.FP32] - terms[sipg.FP64]).max() < 3e-5 * size


@pytest.mark.parametrize("prec,dtype", [(sipg.FP64, np.float64), (sipg.FP32, np.float32)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("dim,n,order", [(2, 4, 2), (2, 5, 1), (3, 2, 3)])
def test_vector_operator_with_slip_faces_in_place(dim, n, order, prec, dtype):
    mesh, t, e, om, x, f, m, bct = random_case(dim, n, order, dim, seed=5 * order + dim, slip=True)
    op = make_op(mesh, order, dim, f, bct=bct)
    xd, yd = DevArray(x.astype(dtype)), DevArray(np.full(x.shape, 7.0, dtype))
    op.apply_device(prec, xd.p, yd.p)
    y = yd.get()
    op.apply_device(prec, xd.p, xd.p)
    assert np.array_equal(xd.get(), y)
