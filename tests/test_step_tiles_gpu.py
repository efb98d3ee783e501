"""Edges of the eight-element tiles of the momentum and projection kernels (meshes below one tile,
whole tiles, a remainder) and device arrays on 8-byte but not 16-byte boundaries, at every order: the device
entries on shifted arrays against the host entries, which the oracle tests cover."""
import ctypes as C

import numpy as np
import pytest

import sipg

pytestmark = pytest.mark.gpu


class Shifted:
    """A device copy of a host array that starts `off` values into its allocation."""

    def __init__(self, host, off):
        self.n, self.off, self.shape = host.size, off, host.shape
        self.v = sipg.DeviceVector(np.concatenate([np.zeros(off), np.asarray(host, np.float64).reshape(-1)]))

    @property
    def p(self):
        return C.c_void_p(self.v.ptr + 8 * self.off)

    def get(self):
        return self.v.get()[self.off:].reshape(self.shape)


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 2, 3])
@pytest.mark.parametrize("off", [0, 1])
def test_advection_on_shifted_arrays(n, order, off):
    mesh = sipg.Mesh.box(3, n, jitter=0.1, seed=3)
    Np = sipg.ref_sizes(3, order)[0]
    rng = np.random.default_rng(order)
    u, uo, no = (rng.uniform(-2, 2, (3, mesh.K, Np)) for _ in range(3))
    bc = rng.integers(0, 3, mesh.Kb).astype(np.int32)
    N, velT = sipg.ins_advection(mesh, order, 1e-3, 2.0, -0.5, 2.0, -1.0, u, uo, no, bc)
    d = [Shifted(x, off) for x in (u, uo, no, np.zeros_like(u), np.zeros_like(u))]
    dbc = sipg.DeviceVector(bc)
    sipg.check(sipg.lib().sipg_ins_advection(
        mesh.h, order, C.c_double(1e-3), C.c_double(2.0), C.c_double(-0.5), C.c_double(2.0), C.c_double(-1.0), d[0].p,
        d[1].p, d[2].p, C.c_void_p(dbc.ptr), d[3].p, d[4].p, C.c_void_p(0)))
    assert np.array_equal(d[3].get(), N) and np.array_equal(d[4].get(), velT)


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("dim,n", [(2, 1), (2, 4), (2, 5), (3, 1), (3, 2), (3, 3)])
@pytest.mark.parametrize("off", [0, 1])
def test_pressure_rhs_on_shifted_arrays(dim, n, order, off):
    mesh = sipg.Mesh.box(dim, n, jitter=0.1, seed=3)
    Np, Nfp, Nf, _ = sipg.ref_sizes(dim, order)
    rng = np.random.default_rng(order)
    v = rng.uniform(-1, 1, (dim, mesh.K, Np))
    dn, do = (rng.uniform(-1, 1, (mesh.K, Nf, Nfp)) for _ in range(2))
    rhs, dold = sipg.pressure_rhs(mesh, order, 1e-2, v, dn, do, 2.0, -1.0)
    d = [Shifted(x, off) for x in (v, dn, do, np.zeros((mesh.K, Np)))]
    sipg.check(sipg.lib().sipg_pressure_rhs(mesh.h, order, C.c_double(1e-2), C.c_double(2.0), C.c_double(-1.0), d[0].p,
                                            d[1].p, d[2].p, d[3].p, C.c_void_p(0)))
    assert np.array_equal(d[3].get(), rhs) and np.array_equal(d[2].get(), dold)


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 2, 3])
@pytest.mark.parametrize("kind", ["grad", "pressure", "two_phase"])
def test_projection_on_shifted_arrays(n, order, kind):
    """Every array shifted alone, and all together: one misaligned pointer takes the unpaired loads."""
    dt = 1e-2
    mesh = sipg.Mesh.box(3, n, jitter=0.1, seed=3)
    Np = sipg.ref_sizes(3, order)[0]
    rng = np.random.default_rng(order)
    v = rng.uniform(-1, 1, (3, mesh.K, Np))
    if kind == "grad":
        ins = [rng.uniform(-1, 1, (3, mesh.K, Np)), v]
        want, st = sipg.project_velocity(mesh, order, dt, *ins)
    else:
        ins = [rng.uniform(-1, 1, (mesh.K, Np)), v]
        rho = rng.uniform(1.0, 1000.0, (mesh.K, Np)) if kind == "two_phase" else None
        want, st = sipg.pressure_projection(mesh, order, dt, *ins, rho=rho)
        if rho is not None:
            ins.insert(1, rho)
    na = len(ins) + 1
    for mask in [0] + [1 << i for i in range(na)] + [(1 << na) - 1]:
        d = [Shifted(x, mask >> i & 1) for i, x in enumerate(ins + [np.zeros_like(v)])]
        dst = sipg.DeviceVector(np.full(2, 12345, np.uint64))
        if kind == "grad":
            sipg.check(sipg.lib().sipg_project_velocity(mesh.h, order, C.c_double(dt), C.c_double(dt), d[0].p, d[1].p,
                                                        d[2].p, C.c_void_p(dst.ptr), C.c_void_p(0)))
        else:
            r = d[1].p if kind == "two_phase" else C.c_void_p(0)
            sipg.check(sipg.lib().sipg_pressure_projection(mesh.h, order, C.c_double(dt), C.c_double(dt), d[0].p, r,
                                                           d[-2].p, d[-1].p, C.c_void_p(dst.ptr), C.c_void_p(0)))
        assert np.array_equal(d[-1].get(), want), mask
        assert dst.get().tolist() == [int(st[1]), int(st[2])], mask
