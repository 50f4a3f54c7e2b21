"""The native linear solve's vector layouts (scalar Jacobian: split by variables; block Jacobian: cell rows) and its chained
launches, at vector lengths of each remainder of 4, with weighted dot products, against the oracle's operators."""
import numpy as np
import pytest
import torch

from dndsr_b200 import mesh as M
from tests.oracle_driver import OracleEval
from tests.test_gpu_linear import _init, _reference_solve, _setup
from tests.util import VR_HQM_PY, relerr

pytestmark = pytest.mark.gpu

# 5 n mod 4: 1, 2, 3, 0
FIVE = [("quad", lambda: M.periodic_quad_2d(7, jitter=0.1), 2, "Roe"), ("tri", lambda: M.periodic_quad_2d(7, jitter=0.1, split_tri=True), 2, "Roe"),
        ("hex", lambda: M.tgv_mesh(3), 3, "Roe"), ("tet", lambda: M.bump_channel_tet(5, 3, 2), 0, "Roe")]
SOLVES = [dict(gmresCode=1, sgsIter=0, nGmresSpace=6, nGmresIter=2), dict(gmresCode=2, sgsIter=1, nGmresSpace=9, nGmresIter=1),
          dict(gmresCode=0, sgsIter=0, nGmresSpace=1, nGmresIter=1)]


def _compare(ev, oe, u0, rhs0, dTau0, kw, scale, modes):
    ref = _reference_solve(oe, u0, rhs0, dTau0, 0.1, 0.5, kw["gmresCode"], 1, kw["sgsIter"], kw["nGmresSpace"], kw["nGmresIter"], meanScale=scale)
    u, rhs, dTau = u0.cuda(), rhs0.cuda(), dTau0.cuda()
    for scalar in modes:
        ev.SetJacobianMode(scalar, False)
        # FP64 and FP32: the bounds of the solve's parity tests
        for prec, tol in (("fp64", 1e-11), ("fp32", 1e-5)):
            x = torch.full_like(rhs, 3.0)
            for _ in range(2):  # the second call replays what the first recorded
                ev.SolveLinear(0.5, dTau, 0.1, u, rhs, x, meanScale=scale, precision=prec, **kw)
            assert relerr(x.cpu().numpy(), ref.numpy()) < tol, (scalar, prec)
    ev.SetJacobianMode(True, False)


@pytest.mark.parametrize("kw", SOLVES, ids=["gmres", "sgs-gmres", "sgs"])
@pytest.mark.parametrize("name,mk,kind,rs", FIVE, ids=[c[0] for c in FIVE])
def test_five_variables(name, mk, kind, rs, kw):
    m, o, vr, ev = _setup(mk, 1, rs, 0.0)
    oe, u0 = OracleEval(o), _init(o, kind)
    dTau0 = torch.zeros(m.n_cell, dtype=torch.float64)
    oe.EvaluateDt(dTau0, u0, 5.0)
    ev.EvaluateDt(torch.zeros(m.n_cell, dtype=torch.float64, device="cuda"), u0.cuda(), 5.0)
    rhs0 = torch.tensor(np.random.default_rng(5).normal(size=(m.n_cell, 5)))
    _compare(ev, oe, u0, rhs0, dTau0, kw, [1.0, 1.2, 1.3, 1.4, 2.5], (True, False))


@pytest.mark.parametrize("kw", SOLVES, ids=["gmres", "sgs-gmres", "sgs"])
@pytest.mark.parametrize("nx", [11, 12])  # 6 n mod 4: 2, 0
def test_six_variables(nx, kw):
    from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction
    from tests.plate_case import plate_oracle, plate_perturbed
    m = M.renumber_by_color(M.flat_plate_hex(nx, 9, 3, y1=1e-3, growth=1.3))
    o, far, mu, types, vals, w = plate_oracle(m, 1, "Roe", 5)
    vr = VariationalReconstruction(m, dict(VR_HQM_PY, maxOrder=1, intOrder=5)).construct(w)
    ev = EulerEvaluator(vr, dict(nVars=6, riemannSolverType="Roe", muGas=mu, muModel=0, prGas=0.72))
    ev.SetBC(types, vals)
    ev.SetWallDistance(M.plate_wall_distance(vr.get("cellPP").reshape(m.n_cell, -1, 3)))
    a, rec = plate_perturbed(m, far, R=o.R)
    oe, u0 = OracleEval(o), torch.tensor(a)
    dTau0 = torch.zeros(m.n_cell, dtype=torch.float64)
    oe.EvaluateDt(dTau0, u0, 5.0)
    u = u0.cuda()
    ev.EvaluateDt(torch.zeros(m.n_cell, dtype=torch.float64, device="cuda"), u, 5.0)
    rhs = torch.zeros_like(u)
    ev.EvaluateRHS(rhs, u, torch.tensor(rec, device="cuda"))  # also the source Jacobian of the diagonal
    r0 = o.eval_rhs(a, rec)
    _compare(ev, oe, u0, torch.tensor(r0), dTau0, kw, [1.0, 1.2, 1.3, 1.4, 2.5, 1.1], (True,))


@pytest.mark.parametrize("name,mk,kind,rs", FIVE, ids=[c[0] for c in FIVE])
def test_block_ilu(name, mk, kind, rs):
    """The tiled block ILU(0): rows in partly filled tiles of 32 and tiles shared by two colours."""
    from tests.test_gpu_roe_jacobian import _reference_solve as reference
    m, o, vr, ev = _setup(mk, 1, rs, 0.0)
    oe, u0 = OracleEval(o), _init(o, kind)
    oe.SetJacobianMode(False, True)
    ev.SetJacobianMode(False, True)
    dTau0 = torch.zeros(m.n_cell, dtype=torch.float64)
    oe.EvaluateDt(dTau0, u0, 5.0)
    u = u0.cuda()
    ev.EvaluateDt(torch.zeros(m.n_cell, dtype=torch.float64, device="cuda"), u, 5.0)
    rec0 = np.zeros((m.n_cell, o.R, 5))
    rhs = torch.zeros_like(u)
    ev.EvaluateRHS(rhs, u, torch.tensor(rec0, device="cuda"))  # also the eigenvalues of the Roe term
    r0 = torch.tensor(o.eval_rhs(u0.numpy(), rec0)) + torch.tensor(np.random.default_rng(5).normal(size=(m.n_cell, 5)))
    for k in (0, 6):  # two ILU steps alone, and as the preconditioner
        ref = reference(oe, u0, r0, dTau0, 0.1, 0.5, int(k > 0), 0, max(k, 1), 1, 2)
        for prec, tol in (("fp64", 1e-10), ("fp32", 1e-5)):  # the bounds of the block solve's parity tests
            x = torch.zeros_like(rhs)
            ev.SolveLinear(0.5, dTau0.cuda(), 0.1, u, r0.cuda(), x, gmresCode=int(k > 0), nGmresSpace=max(k, 1), jacobiCode=2, precision=prec)
            assert relerr(x.cpu().numpy(), ref.numpy()) < tol, (k, prec)
