"""Performance cases of the implicit residual path, through the Python call surface of dndsr_b200.

A case is one pass of work that a user's solver or optimiser repeats:

  residual   EvaluateDt, one VR Jacobi sweep and EvaluateRHS: what every pseudo-iteration does before its
             linear solve (ImplicitSolver.fdtau and frhs)
  linear     EvaluateDt (and EvaluateRHS where the Roe Jacobian needs its eigenvalues) and SolveLinear: the
             linear solve of a pseudo-iteration
  step       a whole ESDIRK4 time step of ImplicitSolver
  vjp        the residual after one VR sweep as a differentiable torch function, forward and backward
  coords     the node-coordinate VJP of the coupled residual, as a shape gradient takes it

on the four flows of the framework's configurations: the isentropic vortex on 2-D triangles or quadrilaterals
(vortex), the Taylor-Green vortex on hexahedra (tgv), the transonic bump in tetrahedra with its boundary zones
(bump) and the SA flat plate on stretched hexahedra (plate).

The mesh, the reconstruction and the evaluator are the plan that a program sets up once: prepare() keeps that of
the last mesh.  States and cotangents come from the seed alone.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from dndsr_b200 import autograd as A
from dndsr_b200 import implicit as I
from dndsr_b200 import mesh as M
from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction, euler_bc_dir_weights

GAMMA = 1.4


def listed():
    return [
        # the smallest call: 8,192 triangles, degree 2, Roe (the isentropic-vortex configuration); launches count
        dict(name="residual-vortex-64", kind="residual", flow="vortex", n=64, tri=True, p=2, flux="Roe"),
        # a whole time step of that configuration: ESDIRK4, 20 pseudo-iterations with one LU-SGS pair per stage
        dict(name="step-vortex-64", kind="step", flow="vortex", n=64, tri=True, p=2, flux="Roe", inner=20),
        # the Taylor-Green configuration and benchmark workload: 262,144 hexahedra, degree 2, HLLE+ and viscous flux
        dict(name="residual-tgv-64", kind="residual", flow="tgv", n=64, p=2, flux="HLLEP"),
        # the steady bump at the size of the derivative configuration: 249,600 tetrahedra, degree 1
        dict(name="residual-bump-250k-p1", kind="residual", flow="bump", nx=80, ny=40, nz=13, p=1, flux="Roe_M2"),
        # the same flow at degree 2 (7 points per face) on an odd mesh
        dict(name="residual-bump-36k-p2", kind="residual", flow="bump", nx=41, ny=21, nz=7, p=2, flux="Roe"),
        # the SA boundary layer: 6 variables, source term, no-slip wall; odd numbers of cells
        dict(name="residual-plate-304k", kind="residual", flow="plate", nx=101, ny=67, nz=45, p=1, flux="Roe"),
        # GMRES(30) with one SGS pair in FP64, the default linear solve of the steady runs
        dict(name="linear-bump-250k-fp64", kind="linear", flow="bump", nx=80, ny=40, nz=13, p=1, flux="Roe_M2", jac="scalar",
             precision="fp64", gmres=30, cfl=200.0),
        # the largest: the steady configuration's 1,996,800 tetrahedra with the FP32 solve inside the defect correction
        dict(name="linear-bump-2m-fp32", kind="linear", flow="bump", nx=160, ny=80, nz=26, p=1, flux="Roe_M2", jac="scalar",
             precision="fp32", gmres=30, cfl=200.0),
        # the Roe Jacobian with the local LU (block ILU(0)) and GMRES(10): the fastest steady settings
        dict(name="linear-roe-250k-fp64", kind="linear", flow="bump", nx=80, ny=40, nz=13, p=1, flux="Roe_M2", jac="roe",
             precision="fp64", gmres=10, cfl=1e4),
        # the derivative configuration: reverse mode of the bump's residual
        dict(name="vjp-bump-250k-p1", kind="vjp", flow="bump", nx=80, ny=40, nz=13, p=1, flux="Roe"),
        # the skin-friction adjoint's operator: reverse mode with the SA model
        dict(name="vjp-plate-77k", kind="vjp", flow="plate", nx=120, ny=80, nz=8, p=1, flux="Roe"),
        # the shape gradient of the pressure drag: node coordinates of the bump mesh
        dict(name="coords-bump-38k-p1", kind="coords", flow="bump", nx=40, ny=20, nz=8, p=1, flux="Roe"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _bump_dims(rng, lo, hi):
    """nx, ny, nz of a channel with about lo to hi tetrahedra, in the proportions of the configurations."""
    s = (math.exp(rng.uniform(math.log(lo), math.log(hi))) / 249600.0) ** (1.0 / 3.0)
    return dict(nx=max(6, int(round(80 * s * rng.uniform(0.9, 1.1)))), ny=max(4, int(round(40 * s * rng.uniform(0.9, 1.1)))),
                nz=max(3, int(round(13 * s * rng.uniform(0.9, 1.1)))))


def draw(rng):
    kind = rng.choice(["residual"] * 4 + ["linear"] * 4 + ["vjp"] * 2 + ["step", "coords"])
    if kind == "step":
        return dict(kind="step", flow="vortex", n=_log_int(rng, 12, 96), tri=rng.random() < 0.5, p=rng.choice([1, 2, 3]), flux="Roe",
                    inner=rng.choice([5, 10, 20]))
    if kind == "coords":
        return dict(kind="coords", flow="bump", **_bump_dims(rng, 1500, 30000), p=1, flux=rng.choice(["Roe", "Roe_M2"]))
    if kind == "linear":
        jac = rng.choice(["scalar", "scalar", "roe"])
        return dict(kind="linear", flow="bump", **_bump_dims(rng, 2000, 400000), p=1, flux="Roe_M2", jac=jac,
                    precision=rng.choice(["fp64", "fp32"]), gmres=rng.choice([5, 10]) if jac == "roe" else rng.choice([0, 10, 30]),
                    cfl=1e4 if jac == "roe" else rng.choice([50.0, 200.0]))
    if kind == "vjp":
        flow = rng.choice(["bump", "plate", "tgv"])
        if flow == "tgv":
            return dict(kind="vjp", flow="tgv", n=_log_int(rng, 8, 40), p=rng.choice([1, 2]), flux="HLLEP")
        if flow == "plate":
            return dict(kind="vjp", flow="plate", nx=rng.randint(24, 120), ny=rng.randint(16, 80), nz=rng.randint(3, 9), p=1, flux="Roe")
        return dict(kind="vjp", flow="bump", **_bump_dims(rng, 2000, 250000), p=rng.choice([1, 2]), flux="Roe")
    flow = rng.choice(["vortex", "tgv", "bump", "plate"])
    if flow == "vortex":
        return dict(kind="residual", flow="vortex", n=_log_int(rng, 12, 256), tri=rng.random() < 0.5, p=rng.choice([1, 2, 3]),
                    flux=rng.choice(["Roe", "HLLEP"]))
    if flow == "tgv":
        return dict(kind="residual", flow="tgv", n=_log_int(rng, 8, 64), p=rng.choice([1, 2]), flux=rng.choice(["HLLEP", "Roe"]))
    if flow == "plate":
        return dict(kind="residual", flow="plate", nx=rng.randint(24, 128), ny=rng.randint(20, 80), nz=_log_int(rng, 3, 40), p=1, flux="Roe")
    p = rng.choice([1, 2])
    return dict(kind="residual", flow="bump", **_bump_dims(rng, 2000, 400000 if p == 1 else 200000), p=p,
                flux=rng.choice(["Roe", "Roe_M2", "HLLC"]))


# ---- the plan: mesh, reconstruction, evaluator ----

class Plan:
    pass


@functools.lru_cache(maxsize=1)
def _plan(key):
    c = dict(key)
    P = Plan()
    hqm = dict(maxOrder=c["p"], dirWeightScheme="HQM_OPT", geomWeightScheme="HQM_SD", geomWeightBias=1.0)
    if c["flow"] == "vortex":
        m = M.periodic_quad_2d(c["n"], L=10.0, jitter=0.1, split_tri=c["tri"])
        vr = VariationalReconstruction(m, dict(hqm, intOrder=5)).construct()
        ev = EulerEvaluator(vr, dict(nVars=5, riemannSolverType=c["flux"], muGas=0.0, ignoreVis=True))
        P.far = np.array([1.0, 1.0, 1.0, 0.0, 1.0 / (GAMMA - 1) + 1.0])
    elif c["flow"] == "tgv":
        m = M.tgv_mesh(c["n"])
        vr = VariationalReconstruction(m, dict(hqm, intOrder=5)).construct()
        ev = EulerEvaluator(vr, dict(nVars=5, riemannSolverType=c["flux"], muGas=1.0 / 1600, muModel=0, prGas=0.71))
        P.far = np.array([1.0, 0.0, 0.0, 0.0, 100.0 / GAMMA / (GAMMA - 1)])
    elif c["flow"] == "bump":
        # the shape gradient is taken on the channel with joined side planes, as its boundary nodes must be off ties
        per = c["kind"] == "coords"
        m = M.bump_channel_tet(c["nx"], c["ny"], c["nz"], periodic_z=per)
        P.far = M.freestream(0.8)
        types, vals = np.zeros(7, np.int32), np.zeros((7, 5))
        for z, t in M.BUMP_BC_TYPES.items():
            if not (per and z > 4):
                types[z], vals[z] = t, P.far
        vr = VariationalReconstruction(m, dict(hqm, intOrder=2 if c["p"] == 1 else 5)).construct(euler_bc_dir_weights(types))
        ev = EulerEvaluator(vr, dict(nVars=5, riemannSolverType=c["flux"], muGas=0.0, ignoreVis=True))
        ev.SetBC(types, vals)
    else:
        m = M.flat_plate_hex(c["nx"], c["ny"], c["nz"], y1=5e-6, growth=1.1)
        far5 = M.freestream(0.2)
        P.mu = np.linalg.norm(far5[1:4]) / far5[0] / 5e6
        P.far = np.concatenate([far5, [3.0 * far5[0]]])
        types, vals, w = np.zeros(6, np.int32), np.zeros((6, 6)), np.ones((6, 4))
        for z, t in M.PLATE_BC_TYPES.items():
            types[z], vals[z], w[z] = t, P.far, (1, 0, 0, 0)
        vr = VariationalReconstruction(m, dict(hqm, intOrder=3)).construct(w)
        ev = EulerEvaluator(vr, dict(nVars=6, riemannSolverType=c["flux"], muGas=P.mu, muModel=0, prGas=0.72))
        ev.SetBC(types, vals)
        ev.SetWallDistance(M.plate_wall_distance(vr.get("cellPP").reshape(m.n_cell, -1, 3)))
    if c.get("jac") == "roe":
        ev.SetJacobianMode(False, True)
    ev.SetDeferredErrors(True)  # as ImplicitSolver does: no synchronisation in every residual
    P.mesh, P.vr, P.ev = m, vr, ev
    P.centre = torch.from_numpy(m.cell_coords().mean(1)).cuda()
    return P


def _plan_of(case):
    # the sizes of a pass (iterations, precision, subspace) are no part of the plan
    return _plan(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "inner", "precision", "gmres", "cfl"))))


# ---- inputs ----

def _waves(x, rng, length):
    """A smooth random field of unit size: five sine waves with periods that fit the length."""
    f = torch.zeros(x.shape[0], dtype=torch.float64, device=x.device)
    for _ in range(5):
        k = torch.from_numpy(rng.integers(-3, 4, size=3) * 2 * np.pi / length).to(x.device)
        f += math.sqrt(0.4) * torch.sin(x @ k + rng.uniform(0, 2 * np.pi))
    return f


def _state(P, case, rng):
    """Cell means of the flow with smooth disturbances of a few per cent."""
    x, flow = P.centre, case["flow"]
    n, nv = x.shape[0], P.ev.nVars
    u = torch.empty((n, nv), dtype=torch.float64, device="cuda")
    if flow in ("vortex", "tgv"):
        P.ev.InitializeUDOF(u, 2 if flow == "vortex" else 3)
        length, amp = (np.array([10.0, 10.0, np.inf]), 0.03) if flow == "vortex" else (np.full(3, 2 * np.pi), 0.01)
    else:
        u[:] = torch.from_numpy(P.far).cuda()
        length, amp = np.array([4.0, 1.0, 0.5]), 0.03
    rho = u[:, 0] * (1 + amp * _waves(x, rng, length))
    v = u[:, 1:4] / u[:, :1]
    p = (GAMMA - 1) * (u[:, 4] - 0.5 * u[:, 0] * (v * v).sum(1)) * (1 + amp * _waves(x, rng, length))
    v = v.clone()
    for d in range(2 if flow == "vortex" else 3):
        v[:, d] += 0.5 * amp * _waves(x, rng, length)
    if flow == "plate":  # a boundary layer over the wall with an eddy viscosity inside it
        y = x[:, 1].clamp_min(0.0) / (0.01 + 0.01 * x[:, 0].clamp_min(0.0))
        v *= torch.where(x[:, 0] > 0, torch.tanh(3 * y), torch.ones_like(y))[:, None]
        u[:, 5] = rho * (3.0 + 60.0 * y * torch.exp(1 - 2 * y) * (1 + amp * _waves(x, rng, length)))
    u[:, 0] = rho
    u[:, 1:4] = rho[:, None] * v
    u[:, 4] = p / (GAMMA - 1) + 0.5 * rho * (v * v).sum(1)
    return u


def _noise(shape, seed, scale):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g) * scale


def prepare(case, seed):
    P = _plan_of(case)
    vr, ev = P.vr, P.ev
    rng = np.random.default_rng([seed, 17])
    S = dict(case=dict(case), plan=P, vr=vr, ev=ev)
    u = S["u"] = _state(P, case, rng)
    nv = ev.nVars
    S["dt"] = torch.zeros(P.mesh.n_cell, dtype=torch.float64, device="cuda")
    if case["kind"] == "linear":
        # a right-hand side of the size of a residual: smooth with some noise
        far = torch.from_numpy(np.abs(P.far) + 0.1).cuda()
        S["rhs"] = _noise(u.shape, seed, 0.2) * far
        for v in range(nv):
            S["rhs"][:, v] += far[v] * _waves(P.centre, rng, np.array([4.0, 1.0, 0.5]))
        S["x"] = torch.zeros_like(u)
        if case["jac"] == "roe":
            S["uRec"], S["res"] = vr.BuildURec(nv), torch.zeros_like(u)
        return S
    # the reconstruction after two sweeps, the running one of a solver that has begun
    a, b = vr.BuildURec(nv), vr.BuildURec(nv)
    vr.DoReconstructionIter(a, b, u, putIntoNew=True)
    vr.DoReconstructionIter(b, a, u, putIntoNew=True)
    S["uRec"] = a
    if case["kind"] == "residual":
        S["uRecNew"], S["rhs"] = b, torch.zeros_like(u)
    elif case["kind"] == "step":
        S["solver"] = I.ImplicitSolver(vr, ev, I.SolverConfig(odeCode=0, dtImplicit=0.01, nTimeStep=1, nTimeStepInternal=case["inner"], CFL=100.0,
                                                              rhsThresholdInternal=0.0, jacobiCode=1, sgsIter=0, gmresCode=0))
        S["out"] = torch.zeros_like(u)
    elif case["kind"] == "vjp":
        u.requires_grad_(True)
        a.requires_grad_(True)
        S["w"] = _noise(u.shape, seed, 1.0)
    else:
        S["w"], S["cot"] = _noise(u.shape, seed, 1.0), _noise(a.shape, seed + 1, 1.0)
    return S


def run(S):
    c, vr, ev, u = S["case"], S["vr"], S["ev"], S["u"]
    if c["kind"] == "residual":
        ev.EvaluateDt(S["dt"], u, 100.0, want_min=False)
        vr.DoReconstructionIter(S["uRec"], S["uRecNew"], u, putIntoNew=True)
        ev.EvaluateRHS(S["rhs"], u, S["uRecNew"])
        return {"dt": S["dt"], "uRec": S["uRecNew"], "rhs": S["rhs"]}
    if c["kind"] == "linear":
        ev.EvaluateDt(S["dt"], u, c["cfl"], want_min=False)
        if c["jac"] == "roe":
            ev.EvaluateRHS(S["res"], u, S["uRec"])
        ev.SolveLinear(1.0, S["dt"], 1e100, u, S["rhs"], S["x"], gmresCode=1 if c["gmres"] else 0, jacobiCode=2 if c["jac"] == "roe" else 1,
                       nGmresSpace=c["gmres"] or 1, precision=c["precision"])
        return S["x"]
    if c["kind"] == "step":
        out, solver = S["out"], S["solver"]
        out.copy_(u)
        solver.uRec.copy_(S["uRec"])
        solver.cfg.res_history.clear()
        solver.run(out)
        return {"u": out, "uRec": solver.uRec}
    if c["kind"] == "vjp":
        ev.EvaluateDt(S["dt"], u, 100.0, want_min=False)
        rhs = A.residual(u, S["uRec"], vr, ev)
        gu, gr = torch.autograd.grad(rhs, (u, S["uRec"]), S["w"])
        return {"rhs": rhs.detach(), "u": gu, "uRec": gr}
    ev.EvaluateDt(S["dt"], u, 100.0, want_min=False)
    return ev.ResidualVJPCoords(S["w"], S["cot"], u, S["uRec"])


# ---- what a pass cannot do without ----

def _sizes(case):
    """cells, faces per cell, dimension, variables, rows of uRec, points per face"""
    p = case["p"]
    if case["flow"] == "vortex":
        return (2 if case["tri"] else 1) * case["n"] ** 2, 3 if case["tri"] else 4, 2, 5, {1: 2, 2: 5, 3: 9}[p], 3
    if case["flow"] == "tgv":
        return case["n"] ** 3, 6, 3, 5, {1: 3, 2: 9}[p], 9
    cells = case["nx"] * case["ny"] * case["nz"]
    if case["flow"] == "bump":
        return 6 * cells, 4, 3, 5, {1: 3, 2: 9}[p], 3 if p == 1 else 7
    return cells, 6, 3, 6, 3, 4


def _residual_work(case):
    nc, nf, d, nv, R, g = _sizes(case)
    visc = case["flow"] in ("tgv", "plate")
    # per cell: uRec and u in, rhs out, barycentre, volume, scales, moments; per face its points; the sweep's matrices
    rhs_b = 8 * ((R + 2) * nv + 2 * d + 1 + R + nf / 2 * (g * (2 * d + 1) + 1))
    vr_b = 8 * (nf * R * (R + 1)) + 8 * (2 * R * nv + nv)
    dt_b = 8 * (nv + 2 + nf / 2 * (d + 1 + 3))
    # per face point: the reconstruction of both sides (values, and gradients where viscous) and the flux
    point = 4 * R * nv * (1 + (d if visc else 0)) + (900 if visc else 450)
    return dict(bytes=nc * (rhs_b + vr_b + dt_b), flops=nc * (nf / 2 * (g * point + 120) + 2 * nf * R * (R + 1) * nv))


def work(case):
    nc, nf, d, nv, R, g = _sizes(case)
    res = _residual_work(case)
    if case["kind"] == "residual":
        return res
    if case["kind"] == "vjp":  # forward, then reverse: the same inputs again, cotangents in place of results
        return dict(bytes=2 * res["bytes"] + nc * 8 * (R + 1) * nv, flops=3.5 * res["flops"])
    if case["kind"] == "coords":
        # every cell's geometry, moments, matrices and fluxes again, and their derivatives to about 8 + nf nodes
        return dict(bytes=nc * 8 * (2 * (R + 1) * nv + 4 * 3 + 2 * (R + 1) + nf * (R + 2)), flops=nc * 3 * 12 * 4000.0)
    if case["kind"] == "step":
        # five implicit stages of `inner` iterations: residual, the update and one SGS pair
        sgs = 8 * (5 * nv + nf / 2 * (d + 2) + 1)
        n = 5 * case["inner"]
        return dict(bytes=n * (res["bytes"] + nc * (2 * sgs + 8 * 6 * nv)), flops=n * (res["flops"] + nc * 160.0 * nf))
    s = 8 if case["precision"] == "fp64" else 4
    k = case["gmres"]
    if case["jac"] == "scalar":
        sweep = s * (3 * nv + nf / 2 * (d + 2) + 1)           # rhs in, x in and out, the faces and the diagonal
        applied, f_app = 2 * sweep, 2 * 75.0 * nf
        product, f_prod = s * (2 * nv + nf / 2 * (d + 2) + 1), 75.0 * nf
    else:
        solve = s * (2 * nv + (nf + 1) * nv * nv)
        product, f_prod = s * (2 * nv + (nf + 1) * nv * nv), 2.0 * nv * nv * (nf + 1)
        applied, f_app = 2 * solve + product, 3 * f_prod       # two LU steps, one product between them
    # Gram-Schmidt reads the basis for the products and for the update, then the solution once more
    gs = s * nv * (k * (k + 1) + 2 * k)
    cells = (k + 1) * applied + k * product + gs + 8 * nv * 3
    flops = (k + 1) * f_app + k * f_prod + 4.0 * nv * k * (k + 1) / 2
    w = dict(bytes=nc * cells, flops=nc * flops)
    if case["jac"] == "roe":
        w = dict(bytes=w["bytes"] + res["bytes"], flops=w["flops"] + res["flops"] + nc * (nf * 1500.0))
    return w


def tolerance(case):
    # Measured: one rounding error in the inputs moves the residual of the Taylor-Green state by 1.1e-12 (it is a
    # difference of fluxes some ten thousand times larger), single entries of the wall cells' cotangents by 7e-12;
    # the FP64 solves are 2e-15 from exact(), the FP32 ones 1.6e-7.
    if case["kind"] == "linear":
        return {"rel": 2e-6, "max": 1e-4} if case["precision"] == "fp32" else {"rel": 1e-13, "max": 1e-12}
    return {"rel": 5e-12, "max": 3e-11}


# ---- the same in plain torch, 64 bits ----

def _t(a, *shape):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda().reshape(*shape)


def _exps(dim, p):
    if dim == 3:
        e = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (0, 1, 1), (1, 0, 1)]
        return e[:{1: 4, 2: 10}[p]]
    e = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (2, 0, 0), (1, 1, 0), (0, 2, 0), (3, 0, 0), (2, 1, 0), (1, 2, 0), (0, 3, 0)]
    return e[:{1: 3, 2: 6, 3: 10}[p]]


class _Torch:
    """The plan's geometry and coefficients as plain tensors, and the operators on them (periodic meshes)."""

    def __init__(self, P, case):
        m, vr = P.mesh, P.vr
        self.case, self.P = case, P
        nf = m.cell2face.shape[1]
        self.c2f = _t(m.cell2face, -1, nf)
        f2c = _t(m.face2cell, -1, 2)
        self.f2c = f2c
        self.side = (f2c[self.c2f, 0] != torch.arange(m.n_cell, device="cuda")[:, None]).long()
        self.nbr = torch.gather(f2c[self.c2f], 2, (1 - self.side)[:, :, None])[:, :, 0]
        self.vol, self.area = _t(vr.get("volume"), -1), _t(vr.get("faceArea"), -1)
        self.mean_n = _t(vr.get("faceMeanNorm"), -1, 3)

    def dt(self, u, cfl):
        """The local time step and, kept for the fluxes and the solve, the face speeds and the jumps' scale."""
        P, c = self.P, self.case
        mu, pr = {"tgv": (1.0 / 1600, 0.71)}.get(c["flow"], (0.0, 0.72))
        i, j = self.f2c[:, 0], self.f2c[:, 1]
        j = torch.where(j < 0, i, j)
        rho, v, p, a = _prim(u)
        vn = (v[i] * self.mean_n).sum(1), (v[j] * self.mean_n).sum(1)
        conv = torch.maximum(a[i] + vn[0].abs(), a[j] + vn[1].abs())
        vis = mu / (0.5 * (rho[i] + rho[j])) * max(4.0 / 3, GAMMA / pr) * self.area * (1 / self.vol[i] + 1 / self.vol[j])
        self.lam = conv + vis
        dvn, da = vn[1] - vn[0], a[j] - a[i]
        jump = torch.maximum(torch.maximum((dvn + da).abs(), (dvn - da).abs()), da.abs())
        self.jump = jump[self.c2f].amax(1)
        ratio = _t(P.vr.get("smoothRatio"), -1)
        return cfl * self.vol * ratio / (self.lam * self.area)[self.c2f].sum(1)

    def sweep(self, uRec, u):
        m, vr = self.P.mesh, self.P.vr
        nf, R = self.c2f.shape[1], uRec.shape[1]
        mat = _t(vr.get("matrixAAInvB"), m.n_cell, nf + 1, R, R)[:, 1:]
        vec = _t(vr.get("vectorAInvB"), m.n_cell, nf, R)
        return torch.einsum("cfij,cfjv->civ", mat, uRec[self.nbr]) + torch.einsum("cfi,cfv->civ", vec, u[self.nbr] - u[:, None])

    def _point(self, side, pts, u, uRec):
        """Values and gradients of one side's reconstruction at the face points."""
        m, vr = self.P.mesh, self.P.vr
        cell = self.f2c[:, side]
        cent, box = _t(vr.get("cellCent"), -1, 3), _t(vr.get("cellHBox"), -1, 3)
        L = box[:, :m.dim].amax(1)
        mom = _t(vr.get("baseMoment"), m.n_cell, -1)
        x = (pts - cent[cell][:, None]) / L[cell][:, None, None]
        ex = _exps(m.dim, self.case["p"])[1:]
        phi = torch.stack([x[..., 0] ** a * x[..., 1] ** b * x[..., 2] ** c for a, b, c in ((*e, 0)[:3] for e in ex)], -1) - mom[cell][:, None, 1:]
        U = u[cell][:, None] + phi @ uRec[cell]
        grads = []
        for d in range(3):
            col = []
            for e in ex:
                e = list((*e, 0)[:3])
                k = e[d]
                e[d] = max(k - 1, 0)
                col.append(k * x[..., 0] ** e[0] * x[..., 1] ** e[1] * x[..., 2] ** e[2])
            grads.append((torch.stack(col, -1) / L[cell][:, None, None]) @ uRec[cell])
        return U, torch.stack(grads, -2)

    def rhs(self, u, uRec):
        m, vr, c = self.P.mesh, self.P.vr, self.case
        pts = _t(vr.get("facePP"), m.n_face, -1, 3)
        n = _t(vr.get("faceNorm"), m.n_face, -1, 3)
        jd = _t(vr.get("faceJDet"), m.n_face, -1)
        w1 = torch.tensor([5.0, 8.0, 5.0], dtype=torch.float64, device="cuda")
        w = w1 if m.dim == 2 else torch.outer(w1, w1).reshape(-1)
        JW = jd * w
        JW = JW * (self.area.sum() / JW.sum())
        sh = _t(m.face_pshift, -1, 3)
        UL, GL = self._point(0, pts, u, uRec)
        UR, GR = self._point(1, pts + sh[:, None], u, uRec)
        i, j = self.f2c[:, 0], self.f2c[:, 1]
        jump = torch.maximum(self.jump[i], self.jump[j])[:, None]
        F = _flux(c["flux"], UL, UR, u[i][:, None], u[j][:, None], n, jump)
        if c["flow"] == "tgv":
            bary = _t(vr.get("cellBary"), -1, 3)
            db = bary[j] - sh - bary[i]
            base = (torch.minimum(self.vol[i], self.vol[j]) * 2 / self.area)[:, None]
            dist = torch.maximum(torch.minimum((n * db[:, None]).sum(-1).abs(), base * 2), base * 0.25)
            G = 0.5 * (GL + GR) + n[..., :, None] * (UR - UL)[..., None, :] / dist[..., None, None]
            F = F - _viscous(0.5 * (UL + UR), G, n, 1.0 / 1600, 0.71)
        total = -(F * JW[..., None]).sum(1)
        sign = 1.0 - 2.0 * self.side
        return (sign[..., None] * total[self.c2f]).sum(1) / self.vol[:, None]


def _prim(U):
    rho = U[..., 0]
    v = U[..., 1:4] / rho[..., None]
    p = (GAMMA - 1) * (U[..., 4] - 0.5 * rho * (v * v).sum(-1))
    return rho, v, p, torch.sqrt(GAMMA * p / rho)


def _physical(U, n):
    rho, v, p, a = _prim(U)
    vn = (v * n).sum(-1)
    F = U * vn[..., None]
    F = torch.cat([F[..., :1], F[..., 1:4] + p[..., None] * n, (F[..., 4] + p * vn)[..., None]], -1)
    return F, vn, a


def _flux(kind, UL, UR, ULm, URm, n, jump):
    """Roe with the Harten-Yee fix, or HLLE+, with the averages of the cell means."""
    FL, _, aL = _physical(UL, n)
    FR, _, aR = _physical(UR, n)
    rl, vl, pl, al = _prim(ULm)
    rr, vr, pr, ar = _prim(URm)
    sl, sr = torch.sqrt(rl), torch.sqrt(rr)
    v = (sl[..., None] * vl + sr[..., None] * vr) / (sl + sr)[..., None]
    H = (sl * (ULm[..., 4] + pl) / rl + sr * (URm[..., 4] + pr) / rr) / (sl + sr)
    v2 = (v * v).sum(-1)
    a = torch.sqrt((GAMMA - 1) * (H - 0.5 * v2))
    vn, vln, vrn = (v * n).sum(-1), (vl * n).sum(-1), (vr * n).sum(-1)
    d = UR - UL
    dn = (d[..., 1:4] * n).sum(-1)
    shear = d[..., 1:4] - d[..., :1] * v
    shear = shear - n * (shear * n).sum(-1)[..., None]
    a1 = (GAMMA - 1) / a ** 2 * (d[..., 0] * (H - vn * vn) + vn * dn - (d[..., 4] - (shear * v).sum(-1)))
    a0 = (d[..., 0] * (vn + a) - dn - a * a1) / (2 * a)
    a4 = d[..., 0] - a0 - a1
    one = torch.ones_like(a1)[..., None]
    if kind == "HLLEP":
        SL, SR = torch.minimum(vn - a, vln - aL), torch.maximum(vn + a, vrn + aR)
        SP, SM = SR.clamp_min(0.0)[..., None], SL.clamp_max(0.0)[..., None]
        fix = a / (a + torch.maximum(vn.abs(), jump.expand_as(vn)))
        wave = torch.cat([one, v.expand(*a1.shape, 3), (0.5 * v2).expand_as(a1)[..., None]], -1)
        return (SP * FL - SM * FR) / (SP - SM) + SP * SM / (SP - SM) * (d - (fix * a1)[..., None] * wave)

    def fixed(lam, ave, left, right):
        t = 0.05 * torch.maximum(torch.maximum(torch.zeros_like(ave), ave - left), right - ave)
        return torch.where(lam < t, (lam * lam / torch.where(t > 0, t, torch.ones_like(t)) + t) * 0.5, lam)

    l0 = fixed((vn - a).abs(), vn - a, vln - al, vrn - ar)
    l1 = fixed(vn.abs(), vn, vln, vrn)
    l4 = fixed((vn + a).abs(), vn + a, vln + al, vrn + ar)
    a0, a1, a4, t = a0 * l0, a1 * l1, a4 * l4, shear * l1[..., None]
    mom = (v - a[..., None] * n) * a0[..., None] + (v + a[..., None] * n) * a4[..., None] + v * a1[..., None] + t
    ene = (H - vn * a) * a0 + 0.5 * v2 * a1 + (H + vn * a) * a4 + (t * v).sum(-1)
    return 0.5 * (FL + FR) - 0.5 * torch.cat([(a0 + a1 + a4)[..., None], mom, ene[..., None]], -1)


def _viscous(U, G, n, mu, pr):
    """The compact viscous flux of the conservative gradient G [..., 3, 5]; Rgas = 1."""
    rho, v, p, _ = _prim(U)
    cp = GAMMA / (GAMMA - 1)
    dv = (G[..., 1:4] - G[..., :1] * v[..., None, :]) / rho[..., None, None]
    dp = (GAMMA - 1) * (G[..., 4] - 0.5 * ((G[..., 1:4] * v[..., None, :]).sum(-1) + (dv * U[..., None, 1:4]).sum(-1)))
    dT = GAMMA / ((GAMMA - 1) * cp) * (dp * rho[..., None] - p[..., None] * G[..., 0]) / rho[..., None] ** 2
    tr = dv[..., 0, 0] + dv[..., 1, 1] + dv[..., 2, 2]
    s = mu * (dv + dv.transpose(-1, -2)) - (2.0 / 3 * mu) * tr[..., None, None] * torch.eye(3, dtype=U.dtype, device=U.device)
    sn = (s * n[..., None, :]).sum(-1)
    e = (sn * v).sum(-1) + cp * mu / pr * (dT * n).sum(-1)
    return torch.cat([torch.zeros_like(e)[..., None], sn, e[..., None]], -1)


def _solve(T, case, u, rhs, dt):
    """LU-SGS pairs and left-preconditioned GMRES on the scalar-Jacobian operator, colour by colour, in 64 bits."""
    n_color, color = T.P.vr.dmesh.colors()
    classes = [torch.from_numpy(np.nonzero(color == k)[0]).cuda() for k in range(n_color)]
    diag = 1 / dt + 0.5 * (T.area * T.lam)[T.c2f].sum(1) / T.vol
    rho, v, p, _ = _prim(u)
    nrm = T.mean_n[T.c2f] * (1.0 - 2.0 * T.side)[..., None]
    w = 0.5 * T.area[T.c2f] / T.vol[:, None] * (T.nbr >= 0)

    def off(cells, x):
        """Sum over the neighbours of w (A(u_o) - lambda) x_o."""
        o, nn = T.nbr[cells].clamp_min(0), nrm[cells]
        U, X, vo, po = u[o], x[o], v[o], p[o]
        dv = (X[..., 1:4] - vo * X[..., :1]) / U[..., :1]
        dp = (GAMMA - 1) * (X[..., 4] - 0.5 * ((X[..., 1:4] * vo).sum(-1) + (U[..., 1:4] * dv).sum(-1)))
        vn, dvn = (vo * nn).sum(-1), (dv * nn).sum(-1)
        F = torch.cat([(X[..., 1:4] * nn).sum(-1)[..., None], X[..., 1:4] * vn[..., None] + U[..., 1:4] * dvn[..., None] + nn * dp[..., None],
                       ((X[..., 4] + dp) * vn + (U[..., 4] + po) * dvn)[..., None]], -1)
        return ((F - T.lam[T.c2f[cells]][..., None] * X) * w[cells][..., None]).sum(1)

    every = torch.arange(u.shape[0], device="cuda")

    def pair(b):
        x = torch.zeros_like(b)
        for k in list(range(n_color)) + list(range(n_color))[::-1]:
            cells = classes[k]
            x[cells] = (b[cells] - off(cells, x)) / diag[cells][:, None]
        return x

    first = pair(rhs)
    k = case["gmres"]
    if not k:
        return first
    beta = first.norm()
    V, H = [first / beta], torch.zeros((k + 1, k), dtype=torch.float64)
    for j in range(k):
        y = pair(diag[:, None] * V[j] + off(every, V[j]))
        h = torch.stack([(y * q).sum() for q in V])
        for hi, q in zip(h, V):
            y = y - hi * q
        H[:j + 1, j], H[j + 1, j] = h.cpu(), y.norm().cpu()
        V.append(y / H[j + 1, j])
    e = torch.zeros((k + 1, 1), dtype=torch.float64)
    e[0] = beta.cpu()
    c = torch.linalg.lstsq(H, e).solution[:, 0]
    return sum(float(ci) * q for ci, q in zip(c, V))


def exact(case, seed):
    """Periodic residuals and their derivatives, and the scalar-Jacobian solves; the rest (ghost states, the SA
    model, block ILU, a hundred pseudo-iterations, second derivatives of the setup) has no short plain form."""
    kind = case["kind"]
    if case["flow"] == "plate" or kind in ("step", "coords") or (kind == "linear" and case["jac"] != "scalar"):
        return None
    S = prepare(case, seed)
    T = _Torch(S["plan"], case)
    u = S["u"].detach()
    dt = T.dt(u, case.get("cfl", 100.0))
    if kind == "linear":
        return _solve(T, case, u, S["rhs"], dt)
    if case["flow"] == "bump":
        return {"dt": dt, "uRec": None, "rhs": None} if kind == "residual" else None
    u, r0 = u.clone().requires_grad_(kind == "vjp"), S["uRec"].detach().clone().requires_grad_(kind == "vjp")
    uRec = T.sweep(r0, u)
    rhs = T.rhs(u, uRec)
    if kind == "residual":
        return {"dt": dt, "uRec": uRec, "rhs": rhs}
    gu, gr = torch.autograd.grad(rhs, (u, r0), S["w"])
    return {"rhs": rhs.detach(), "u": gu, "uRec": gr}
