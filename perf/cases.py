"""Performance cases: the work a user of this library has it do, through its public entry points.

Kinds (a case is a dict of plain values; every mesh is a box of simplices with vertices
jittered by 0.1 h, inputs come from the seed):

  apply       one operator application on device vectors (Operator.apply_device), 2D and 3D,
              orders 1-4, FP32 (TF32 tensor cores) and FP64: constant, two-phase (1 / rho,
              density ratio 1000) and Helmholtz coefficients, scalar or the coupled vector
              operator with slip walls
  solve       one linear solve from a zero guess (Solver.solve_device), the set-up done
              beforehand: p-multigrid in mixed or FP64 precision, block-Jacobi PCG, and the
              Jacobi PCG of the coupled viscous operator
  refactor    a pressure solve of a time step whose density moved: new nodal factor, solver
              set-up, solve (Operator.set_factor, Solver.setup, Solver.solve_device)
  projection  pressure gradient and velocity projection (sipg_pressure_projection)
  momentum    the kernels before the pressure solve: advection, pressure Neumann data,
              pressure right-hand side (sipg_ins_advection, sipg_ins_pressure_neumann,
              sipg_pressure_rhs)
  bubble      the two-phase time step as a whole: initial state with its level-set
              reinitialisation, a few steps, the fields back to the host (Ins3D)
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ins-solver_b200"))
import sipg  # noqa: E402

MAX_DOF = 23.3e6  # the largest listed vector: 48^3 x 6 tets at p = 4


def listed():
    return [
        # a small 2D problem's operator: the smallest call, launches and latency
        dict(name="apply_2d_small", kind="apply", dim=2, n=23, order=2, bits=32, coef="const", ncomp=1),
        # the V-cycle's fine-level apply at the headline pressure problem's size
        dict(name="apply_p3_f32", kind="apply", dim=3, n=24, order=3, bits=32, coef="two_phase", ncomp=1),
        # the large Helmholtz configuration, FP64
        dict(name="apply_p4_f64", kind="apply", dim=3, n=48, order=4, bits=64, coef="helmholtz", ncomp=1),
        # a small served Poisson problem in full precision: latency of the multigrid loop
        dict(name="solve_small_f64", kind="solve", solver="pmg", dim=3, n=7, order=3, bits=64, coef="const"),
        # 2D manufactured-Poisson configuration: block-Jacobi PCG to 1e-10
        dict(name="solve_2d_blockjacobi", kind="solve", solver="block_jacobi", dim=2, n=64, order=3, bits=64,
             coef="const"),
        # the headline pressure solve: two-phase factor, mixed-precision p-multigrid
        dict(name="solve_pressure_mixed", kind="solve", solver="pmg", dim=3, n=24, order=3, bits=32,
             coef="two_phase"),
        # the viscous step's coupled solve with slip walls: Jacobi PCG on (u, v, w)
        dict(name="solve_viscous", kind="solve", solver="viscous", dim=3, n=16, order=3, bits=64, coef="viscous"),
        # one time step's pressure solve after the density moved, p = 4, odd size
        dict(name="refactor_p4", kind="refactor", dim=3, n=13, order=4, bits=32, coef="two_phase"),
        # velocity projection after the pressure solve at the rising-bubble size
        dict(name="projection_p3", kind="projection", dim=3, n=32, order=3, rho=True),
        # advection and pressure right-hand side at the rising-bubble size
        dict(name="momentum_p3", kind="momentum", n=32, order=3),
        # a short full-precision two-phase run on a coarse mesh with an open top
        dict(name="bubble_small", kind="bubble", n=8, order=2, bits=64, over_int=False, steps=4, walls="open"),
        # the rising bubble: over-integrated pressure, mixed p-multigrid
        dict(name="bubble", kind="bubble", n=24, order=3, bits=32, over_int=True, steps=4, walls="closed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same ranges."""
    kind = rng.choice(["apply", "apply", "solve", "solve", "refactor", "projection", "momentum", "bubble"])
    if kind == "apply":
        dim, order = rng.choice([2, 3, 3]), rng.randint(1, 4)
        ncomp = rng.choice([1, 1, 1, dim]) if dim == 3 else 1
        coef = "viscous" if ncomp > 1 else rng.choice(["const", "two_phase", "helmholtz"])
        cap = MAX_DOF / ncomp / sipg_np(dim, order)
        top = int((cap / 2) ** 0.5) if dim == 2 else int((cap / 6) ** (1.0 / 3.0))
        n = _log_int(rng, 12, min(600, top)) if dim == 2 else _log_int(rng, 3, min(48, top))
        return dict(kind=kind, dim=dim, n=n, order=order, bits=rng.choice([32, 64]), coef=coef, ncomp=ncomp)
    if kind == "solve":
        solver = rng.choice(["pmg", "pmg", "pmg", "block_jacobi", "viscous"])
        if solver == "pmg":
            dim = rng.choice([2, 3])
            n = _log_int(rng, 24, 160) if dim == 2 else _log_int(rng, 5, 24)
            order = rng.randint(2, 3 if dim == 3 and n > 18 else 4)
            return dict(kind=kind, solver=solver, dim=dim, n=n, order=order, bits=rng.choice([32, 32, 64]),
                        coef=rng.choice(["const", "two_phase"]))
        if solver == "block_jacobi":
            return dict(kind=kind, solver=solver, dim=2, n=_log_int(rng, 12, 64), order=rng.randint(1, 4), bits=64,
                        coef="const")
        return dict(kind=kind, solver=solver, dim=3, n=_log_int(rng, 4, 16), order=rng.randint(1, 3), bits=64,
                    coef="viscous")
    if kind == "refactor":
        return dict(kind=kind, dim=3, n=_log_int(rng, 5, 18), order=rng.randint(2, 4), bits=rng.choice([32, 32, 64]),
                    coef="two_phase")
    if kind == "projection":
        dim, order = rng.choice([2, 3, 3]), rng.randint(1, 4)
        n = _log_int(rng, 16, 256) if dim == 2 else _log_int(rng, 4, 32 if order < 4 else 24)
        return dict(kind=kind, dim=dim, n=n, order=order, rho=rng.random() < 0.7)
    if kind == "momentum":
        order = rng.randint(1, 4)
        return dict(kind=kind, n=_log_int(rng, 4, 32 if order < 4 else 24), order=order)
    return dict(kind=kind, n=_log_int(rng, 6, 18), order=rng.randint(2, 3), bits=rng.choice([32, 64]),
                over_int=rng.random() < 0.5, steps=rng.randint(2, 4), walls=rng.choice(["closed", "open", "slip"]))


def sipg_np(dim, p):
    return (p + 1) * (p + 2) // 2 if dim == 2 else (p + 1) * (p + 2) * (p + 3) // 6


def _cells(c):
    return 2 * c["n"] ** 2 if c.get("dim", 3) == 2 else 6 * c["n"] ** 3


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(shape, seed, lo=-1.0, hi=1.0, dtype=torch.float64):
    return (torch.rand(shape, dtype=torch.float64, device="cuda", generator=_gen(seed)) * (hi - lo) + lo).to(dtype)


def _nodes(e):
    """Node coordinates (dim, K, Np) on the GPU."""
    return torch.stack([torch.from_numpy(e[k]).cuda() for k in ("x", "y", "z")[:e["dim"]]])


def _smooth_step(nodes, n, ratio, radius=0.25, width=1.5):
    """1 outside and `ratio` inside a ball at the centre, smoothed by tanh over 1.5 h."""
    r = torch.sqrt(((nodes - 0.5) ** 2).sum(0))
    return 1.0 + (ratio - 1.0) * 0.5 * (1.0 + torch.tanh((radius - r) * n / width))


def _radius(seed):
    return 0.2 + 0.1 * float(np.random.default_rng(int(seed)).random())


def _rhs(mesh_e, t, nodes, seed, mean_free, modes=32):
    """J M f of a Gaussian random field f with correlation length 0.1 (random Fourier
    modes), its mean removed for the Neumann problems."""
    g = _gen(seed + 1)
    k = torch.randn((modes, mesh_e["dim"]), dtype=torch.float64, device="cuda", generator=g) / 0.1
    ph = torch.rand((modes,), dtype=torch.float64, device="cuda", generator=g) * (2 * math.pi)
    f = torch.zeros_like(nodes[0])
    for i in range(modes):
        f += torch.cos(torch.tensordot(k[i], nodes, 1) + ph[i])
    f *= math.sqrt(2.0 / modes)
    J, M = torch.from_numpy(mesh_e["geof"][:, -1].copy()).cuda(), torch.from_numpy(t["M"]).cuda()
    mass = lambda v: J[:, None] * (v @ M.T)  # noqa: E731
    if mean_free:
        f = f - mass(f).sum() / mass(torch.ones_like(f)).sum()
    return mass(f)


def _operator(c, seed):
    """Mesh, operator and what defines it (host boundary types, coefficients on the GPU)."""
    dim, n, order, coef = c["dim"], c["n"], c["order"], c["coef"]
    mesh = sipg.Mesh.box(dim, n, jitter=0.1, seed=int(seed) & 0x7FFFFFFF)
    ncomp = dim if coef == "viscous" else 1
    op = sipg.Operator(mesh, order, ncomp)
    d = dict(mesh=mesh, op=op, factor=None, mm=None, mm_scalar=0.0, ncomp=ncomp)
    if coef in ("two_phase", "viscous"):
        e = mesh.export(order)
        nodes = _nodes(e)
        d.update(e=e, nodes=nodes)
    if coef == "const":  # zero Dirichlet walls (the manufactured problem), Neumann for p-multigrid
        neumann = c.get("solver") == "pmg"
        d["bct"] = np.full((1, mesh.Kb), sipg.BC_NEUMANN if neumann else sipg.BC_DIRICHLET, np.int32)
    elif coef == "two_phase":
        d["bct"] = np.full((1, mesh.Kb), sipg.BC_NEUMANN, np.int32)
        d["factor"] = 1.0 / _smooth_step(nodes, n, 1000.0, _radius(seed))
    elif coef == "helmholtz":  # I / (nu dt) - Laplacian, nu = dt = 1e-3
        d["bct"] = np.full((1, mesh.Kb), sipg.BC_DIRICHLET, np.int32)
        d["mm_scalar"] = 1e6
    else:  # the viscous step: mu-weighted operator + g0 Re rho / dt mass, slip x / z walls
        yb = e["bface_centroid"][:, 1]
        wall = np.where((yb < 1e-9) | (yb > 1 - 1e-9), sipg.BC_DIRICHLET, sipg.BC_SLIP).astype(np.int32)
        d["bct"] = np.repeat(wall[None], ncomp, axis=0)
        rad = _radius(seed)
        d["factor"] = _smooth_step(nodes, n, 100.0, rad)
        d["mm"] = 1.5 * 100.0 / 1e-3 * _smooth_step(nodes, n, 1000.0, rad)
    op.set_bc_types(d["bct"])
    if d["factor"] is not None:
        op.set_factor(d["factor"].cpu().numpy())
    if d["mm"] is not None:
        op.set_mm(sipg.MM_NODAL, 0.0, d["mm"].cpu().numpy())
    elif d["mm_scalar"]:
        op.set_mm(sipg.MM_SCALAR, d["mm_scalar"])
    return d


def _solver(c, op):
    if c.get("solver", "pmg") == "pmg":
        o = sipg.default_opts(sipg.SOLVER_PMULTIGRID)
        o.precision = c["bits"]
        o.n_levels = c["order"]
        for lev in range(4):
            o.orders[lev] = max(0, c["order"] - lev)
        o.rel_tol, o.abs_tol, o.nullspace = 1e-8, 0.0, 1
        return sipg.Solver(op, sipg.SOLVER_PMULTIGRID, o)
    kind = sipg.SOLVER_BLOCK_JACOBI if c["solver"] == "block_jacobi" else sipg.SOLVER_JACOBI
    o = sipg.default_opts(kind)
    o.rel_tol, o.abs_tol, o.max_iter = (1e-10 if c["solver"] == "block_jacobi" else 1e-8), 0.0, 5000
    return sipg.Solver(op, kind, o)


def _system(c, seed):
    """Operator, right-hand side, solution vector and a solver that is set up."""
    s = _operator(c, seed)
    e = s.setdefault("e", s["mesh"].export(c["order"]))
    nodes = s.setdefault("nodes", _nodes(e))
    t = sipg.ref_tables(c["dim"], c["order"])
    b = torch.stack([_rhs(e, t, nodes, seed + 7 * comp, c.get("solver", "pmg") == "pmg")
                     for comp in range(s["ncomp"])])
    s.update(b=b, x=torch.zeros_like(b), solver=_solver(c, s["op"]))
    s["solver"].setup()
    return s


def prepare(case, seed):
    c = case
    kind = c["kind"]
    if kind == "apply":
        s = _operator(c, seed)
        dt = torch.float32 if c["bits"] == 32 else torch.float64
        s["x"] = _uniform(s["op"].shape(), seed, dtype=dt)
        s["y"] = torch.empty_like(s["x"])
    elif kind in ("solve", "refactor"):
        s = _system(c, seed)
        if kind == "refactor":  # the density after the interface moved
            s["new_factor"] = (1.0 / _smooth_step(s["nodes"], c["n"], 1000.0, _radius(seed) + 0.01)).cpu().numpy()
    elif kind == "projection":
        mesh = sipg.Mesh.box(c["dim"], c["n"], jitter=0.1, seed=int(seed) & 0x7FFFFFFF)
        shape = (mesh.K, sipg_np(c["dim"], c["order"]))
        s = dict(mesh=mesh, pr=_uniform(shape, seed), velT=_uniform((c["dim"],) + shape, seed + 1))
        s["rho"] = _uniform(shape, seed + 2, 1.0, 1000.0) if c["rho"] else None
        s["out"] = torch.empty_like(s["velT"])
    elif kind == "momentum":
        mesh = sipg.Mesh.box(3, c["n"], jitter=0.1, seed=int(seed) & 0x7FFFFFFF)
        Np, Nfp = sipg.ref_sizes(3, c["order"])[:2]
        v = (3, mesh.K, Np)
        s = dict(mesh=mesh, u=_uniform(v, seed), u_old=_uniform(v, seed + 1), N_old=_uniform(v, seed + 2),
                 mu=_uniform(v[1:], seed + 3, 0.01, 1.0), rho=_uniform(v[1:], seed + 4, 0.001, 1.0))
        s["bc"] = torch.randint(0, 3, (mesh.Kb,), dtype=torch.int32, device="cuda", generator=_gen(seed + 5))
        s.update(N=torch.empty(v, dtype=torch.float64, device="cuda"),
                 velT=torch.empty(v, dtype=torch.float64, device="cuda"),
                 dPdN=torch.empty((mesh.K, 4, Nfp), dtype=torch.float64, device="cuda"),
                 rhs=torch.empty(v[1:], dtype=torch.float64, device="cuda"))
    else:
        mesh = sipg.Mesh.box(3, c["n"], jitter=0.1, seed=int(seed) & 0x7FFFFFFF)
        e = mesh.export(c["order"])
        r = np.random.default_rng(int(seed)).uniform(-1.0, 1.0, 4)
        ball = np.sqrt((e["x"] - 0.5 - 0.05 * r[0]) ** 2 + (e["y"] - 0.3 - 0.05 * r[1]) ** 2
                       + (e["z"] - 0.5 - 0.05 * r[2]) ** 2) - 0.25 - 0.03 * r[3]
        bc = np.zeros(mesh.Kb, np.int32)  # no-slip walls
        if c["walls"] == "open":  # natural outflow at the top
            bc[e["bface_centroid"][:, 1] > 1 - 1e-9] = 2
        elif c["walls"] == "slip":
            bc[(e["bface_centroid"][:, 0] < 1e-9) | (e["bface_centroid"][:, 0] > 1 - 1e-9)] = 1
        ins = sipg.Ins3D(mesh, bc, order=c["order"], reynolds=100.0, rho0=1.0, rho1=1e-3, mu0=1.0, mu1=1e-2,
                         gravity=9.81, cfl=0.5, pr_over_int=int(c["over_int"]), precision=c["bits"])
        s = dict(ins=ins, vel=np.zeros((3,) + ball.shape), ls=ball)
    s["case"] = dict(c)
    return s


# ------------------------------------------------------------------ one pass
_P, _D = ctypes.c_void_p, ctypes.c_double


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    stream = torch.cuda.current_stream()
    if kind == "apply":
        s["op"].apply_device(c["bits"], s["x"].data_ptr(), s["y"].data_ptr(), stream.cuda_stream)
        return s["y"]
    if kind in ("solve", "refactor"):
        s["x"].zero_()
        if kind == "refactor":
            s["op"].set_factor(s["new_factor"])
            s["solver"].setup()
        stream.synchronize()  # the solver runs on its own stream
        s["solver"].solve_device(s["b"].data_ptr(), s["x"].data_ptr())
        return s["x"]
    if kind == "projection":
        dt = 1e-3
        sipg.check(sipg.lib().sipg_pressure_projection(
            s["mesh"].h, c["order"], _D(dt), _D(sipg.projection_factor(c["dim"], dt)), _P(s["pr"].data_ptr()),
            _P(s["rho"].data_ptr() if s["rho"] is not None else 0), _P(s["velT"].data_ptr()),
            _P(s["out"].data_ptr()), _P(0), _P(stream.cuda_stream)))
        return s["out"]
    if kind == "momentum":
        p = {k: _P(s[k].data_ptr()) for k in ("u", "u_old", "N_old", "bc", "mu", "rho", "N", "velT", "dPdN", "rhs")}
        h, o, st, lib = s["mesh"].h, c["order"], _P(stream.cuda_stream), sipg.lib()
        a0, a1, b0, b1 = 2.0, -0.5, 2.0, -1.0
        sipg.check(lib.sipg_ins_advection(h, o, _D(1e-3), _D(a0), _D(a1), _D(b0), _D(b1), p["u"], p["u_old"],
                                          p["N_old"], p["bc"], p["N"], p["velT"], st))
        sipg.check(lib.sipg_ins_pressure_neumann(h, o, _D(100.0), p["u"], p["N"], p["mu"], p["rho"], p["bc"],
                                                 p["dPdN"], st))
        sipg.check(lib.sipg_pressure_rhs(h, o, _D(1e-3), _D(b0), _D(0.0), p["velT"], p["dPdN"], _P(0), p["rhs"], st))
        return {k: s[k] for k in ("N", "velT", "dPdN", "rhs")}
    s["ins"].set_state(s["vel"], s["ls"])
    s["ins"].step(c["steps"])
    return s["ins"].state()


# ------------------------------------------------------------------ accounting
def work(case):
    """Bytes: each input and output once (vectors, coefficients, geometric factors, face
    neighbours). Flops: the contractions of the operator's definition once; of a solve or a
    time step one operator application (the iterations are the method's)."""
    c = case
    dim, p = c.get("dim", 3), c["order"]
    K, Np, Nf = _cells(c), sipg_np(dim, p), dim + 1
    Nfp = p + 1 if dim == 2 else (p + 1) * (p + 2) // 2
    w = 4 if c.get("bits") == 32 and c["kind"] == "apply" else 8
    geo = (dim * dim + 1) * w + 8 * Nf
    mult = 2 * (2 * dim + 1) * Np * Np + 2 * (dim + 1) * Np * Nf * Nfp
    if c["kind"] == "apply" or c["kind"] in ("solve", "refactor"):
        nc = dim if c["coef"] == "viscous" else 1
        coefs = {"const": 0, "helmholtz": 0, "two_phase": 1, "viscous": 2}[c["coef"]]
        return dict(bytes=K * (Np * w * (2 * nc + coefs) + geo), flops=K * nc * mult)
    if c["kind"] == "projection":
        return dict(bytes=K * (8 * Np * (2 * dim + 1 + int(c["rho"])) + geo),
                    flops=K * (2 * Np * Np * (3 * dim + 2) + 2 * Np * Nf * Nfp))
    if c["kind"] == "momentum":
        return dict(bytes=K * (8 * Np * (3 * 5 + 1 + 2) + 8 * Nf * Nfp + geo),
                    flops=K * (2 * Np * Np * (9 + 3 + 1) + 2 * Np * Nf * Nfp * 5))
    return dict(bytes=K * (8 * Np * (4 + 7) + geo) * c["steps"], flops=K * mult * 4 * c["steps"])


def tolerance(case):
    c = case
    if c["kind"] == "apply":
        if c["bits"] == 64:
            return dict(rel=1e-13, max=1e-11)
        # TF32 operands (10 mantissa bits): 4e-4 to 7e-4 from the FP64 result
        return dict(rel=3e-3, max=0.2)
    if c["kind"] in ("solve", "refactor"):
        # each stops at a relative residual of 1e-8 (block Jacobi 1e-10); against a solve to 1e-13
        # their solutions are off by up to 6e-12 (block Jacobi), 3e-10 (p-multigrid) and 8e-8 (viscous)
        if c.get("solver") == "viscous":
            return dict(rel=4e-7, max=2e-5)
        return dict(rel=1e-10, max=1e-8) if c.get("solver") == "block_jacobi" else dict(rel=4e-9, max=2e-7)
    if c["kind"] == "projection":
        # the element solves stop at an absolute residual of 1e-8 (2D: |r|^2 < 1e-16 of an
        # unpreconditioned system scaled by h^2, which leaves more of the round-off in)
        return dict(rel=1e-10, max=1e-8) if c["dim"] == 3 else dict(rel=1e-3, max=0.2)
    if c["kind"] == "momentum":
        return dict(rel=1e-13, max=1e-11)
    # the viscous solves' 1e-8: velocities are up to 1.4e-7 (largest 1.6e-5 of the r.m.s.) from a
    # run whose solves go to 1e-12
    return dict(rel=6e-7, max=6e-5)


# ------------------------------------------------------------------ 64-bit answers
class _Disc:
    """Tables and face pairing of a mesh on the GPU, for plain torch in FP64. The nodes,
    derivative and mass tables and the face pairing define the discretisation (they are data of
    the problem); every operation on them below is torch's."""

    def __init__(self, mesh, dim, order):
        e, t = mesh.export(order), sipg.ref_tables(dim, order)
        self.dim, self.K, self.Np, self.Nf, self.Nfp = dim, e["K"], e["Np"], e["Nf"], e["Nfp"]
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        self.D = [up(t[k]) for k in ("Dr", "Ds", "Dt")[:dim]]
        self.M, self.E = up(t["M"]), up(t["EMAT"])
        self.LIFT = torch.linalg.solve(self.M, self.E)
        self.fm = up(t["fmask"].astype(np.int64))
        geof = up(e["geof"])
        self.J, self.G = geof[:, -1], geof[:, :dim * dim].reshape(-1, dim, dim)  # G[e][r][d] = dr_r / dx_d
        self.n = torch.stack([up(e[k]) for k in ("nx", "ny", "nz")[:dim]])        # dim x K x Nf
        self.sJ, self.fs = up(e["sJ"]), up(e["fscale"])
        K, Np, Nf = self.K, self.Np, self.Nf
        ext = np.full((K, Nf, Np), -1, np.int64)
        nbf = np.full((K, Nf), -1, np.int64)
        L, R = e["face2cells"].T.astype(np.int64)
        fL, fR = e["faceNum"].T
        ext[L[:, None], fL[:, None], e["fmaskL"]] = R[:, None] * Np + e["fmaskR"]
        ext[R[:, None], fR[:, None], e["fmaskR"]] = L[:, None] * Np + e["fmaskL"]
        nbf[L, fL], nbf[R, fR] = R * Nf + fR, L * Nf + fL
        ext = np.stack([ext[:, f][:, t["fmask"][f]] for f in range(Nf)], 1)
        self.ext, self.nbf = up(ext), up(nbf)  # neighbour's node of each face node, neighbour's face
        self.inner = self.nbf >= 0
        bf = np.full((K, Nf), 0, np.int64)
        bf[e["bface2cell"], e["bfaceNum"]] = np.arange(e["Kb"])
        self.bf = up(bf)

    def own(self, v):
        return v[..., self.fm]

    def other(self, v):
        """The neighbour's value at each face node (own value on boundary faces)."""
        w = v.reshape(v.shape[:-2] + (-1,))[..., self.ext.clamp(min=0)]
        return torch.where(self.inner[..., None], w, self.own(v))

    def grad(self, v):
        dr = [v @ D.T for D in self.D]
        return torch.stack([sum(self.G[:, r, d, None] * dr[r] for r in range(self.dim)) for d in range(self.dim)])

    def lift(self, f):
        return f.reshape(f.shape[:-2] + (-1,)) @ self.LIFT.T

    def emat(self, f):
        return f.reshape(f.shape[:-2] + (-1,)) @ self.E.T


def _exact_apply(c, s, x):
    g, dim = _Disc(s["mesh"], c["dim"], c["order"]), c["dim"]
    f = s["factor"] if s["factor"] is not None else torch.ones((g.K, g.Np), dtype=torch.float64, device="cuda")
    p = c["order"]
    fown, foth = g.own(f), g.other(f)
    fs_other = torch.where(g.inner, g.fs.reshape(-1)[g.nbf.clamp(min=0)], g.fs)
    tau = 2.0 * (p + 1) * (p + 2) * torch.maximum(g.fs[..., None] * fown, fs_other[..., None] * foth).amax(-1)
    bct = torch.from_numpy(s["bct"]).cuda()
    nc = s["ncomp"]
    um = [g.own(x[k]) for k in range(nc)]
    q = [f * g.grad(x[k]) for k in range(nc)]
    nq = [sum(g.n[d, ..., None] * g.own(q[k][d]) for d in range(dim)) for k in range(nc)]
    ys = []
    for k in range(nc):
        jump = um[k] - g.other(x[k])
        nqo = sum(g.n[d, ..., None] * g.other(q[k][d]) for d in range(dim))
        navg = 0.5 * (nq[k] + nqo)
        kind = torch.where(g.inner, torch.full_like(g.bf, -1), bct[k][g.bf].long())[..., None]
        jump = torch.where(kind == sipg.BC_DIRICHLET, 2 * um[k], jump)
        navg = torch.where(kind == sipg.BC_DIRICHLET, nq[k], navg)
        jump = torch.where(kind == sipg.BC_NEUMANN, torch.zeros_like(jump), jump)
        navg = torch.where(kind == sipg.BC_NEUMANN, torch.zeros_like(jump), navg)
        if nc > 1:  # slip walls: the normal component is a Dirichlet one
            un = sum(g.n[d, ..., None] * um[d] for d in range(nc))
            nnq = sum(g.n[d, ..., None] * nq[d] for d in range(nc))
            jump = torch.where(kind == sipg.BC_SLIP, 2 * g.n[k, ..., None] * un, jump)
            navg = torch.where(kind == sipg.BC_SLIP, g.n[k, ..., None] * nnq, navg)
        fu = g.sJ[..., None] * (0.5 * tau[..., None] * jump - navg)
        sv = -0.5 * g.sJ[..., None] * fown * jump
        y = g.emat(fu)
        for r in range(dim):
            vol = g.J[:, None] * sum(g.G[:, r, d, None] * q[k][d] for d in range(dim))
            cr = sum(g.G[:, r, d, None] * g.n[d] for d in range(dim))
            y = y + (vol @ g.M.T + g.emat(cr[..., None] * sv)) @ g.D[r]
        mm = s["mm"] if s["mm"] is not None else s["mm_scalar"]
        y = y + g.J[:, None] * ((mm * x[k]) @ g.M.T)
        ys.append(y)
    return torch.stack(ys)


def _exact_momentum(c, s):
    g, dt = _Disc(s["mesh"], 3, c["order"]), 1e-3
    u, n = s["u"], g.n[..., None]
    uM, uP = g.own(u), g.other(u)
    kind = torch.where(g.inner, torch.full_like(g.bf, -1), s["bc"].long()[g.bf])[..., None]
    lvel = (n * uM).sum(0)
    uP = torch.where(kind == 0, torch.zeros_like(uP), torch.where(kind == 1, uM - n * lvel, uP))
    rvel = (n * uP).sum(0)
    lam = torch.maximum(lvel.abs(), rvel.abs())
    lam = torch.where(g.inner[..., None], lam, lam.amax(-1, keepdim=True).floor())
    flux = 0.5 * g.fs[..., None] * (-(uM * lvel - uP * rvel) - lam * (uP - uM))
    div = lambda F: sum(g.G[:, r, d, None] * (F[d] @ g.D[r].T) for r in range(3) for d in range(3))  # noqa: E731
    N = torch.stack([div(u[k] * u) + g.lift(flux[k]) for k in range(3)])
    velT = 2.0 * u - 0.5 * s["u_old"] - dt * (2.0 * N - s["N_old"])

    def curl(v):
        d = [g.grad(v[k]) for k in range(3)]
        return torch.stack([d[2][1] - d[1][2], d[0][2] - d[2][0], d[1][0] - d[0][1]])
    res = -N - curl(s["mu"] * curl(u)) / (100.0 * s["rho"])
    dPdN = torch.where((kind == 0) | (kind == 1), g.fs[..., None] * (n * g.own(res)).sum(0), torch.zeros_like(lvel))
    half = 0.5 * g.fs[..., None] * (n * (g.other(velT) - g.own(velT))).sum(0)
    rhs = g.J[:, None] * ((-(div(velT) + g.lift(half)) / dt + 2.0 * g.lift(dPdN)) @ g.M.T)
    return dict(N=N, velT=velT, dPdN=dPdN, rhs=rhs)


def exact(case, seed):
    """What run() returns, in plain FP64 torch. None for the solves, the projection and the time
    steps: their answers are those of an iteration stopped at a residual (the projection's at an
    absolute one that leaves up to a percent), not a closed formula's."""
    if case["kind"] == "apply":
        s = prepare(case, seed)
        return _exact_apply(case, s, s["x"].double())
    if case["kind"] == "momentum":
        return _exact_momentum(case, prepare(case, seed))
    return None
