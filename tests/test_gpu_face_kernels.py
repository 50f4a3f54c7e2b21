"""The inviscid face kernels (cell rows staged by the warps) at ragged face counts and each quadrature size that they cover,
with periodic, interior and boundary faces: the residual against the oracle, the transpose against the tangent."""
import numpy as np
import pytest
import torch

from dndsr_b200 import mesh as M
from tests.bump_case import bump_oracle, perturbed_state
from tests.util import VR_HQM_PY, relerr

pytestmark = pytest.mark.gpu

# name, mesh (None: the bump channel), degree, quadrature order, Riemann solver
CASES = [("tri-p1-o1", lambda: M.periodic_quad_2d(5, jitter=0.1, split_tri=True), 1, 1, "Roe"),
         ("tri-p1-o5", lambda: M.periodic_quad_2d(7, jitter=0.1, split_tri=True), 1, 5, "HLLEP"),
         ("quad-p2-o3", lambda: M.periodic_quad_2d(7, jitter=0.1), 2, 3, "Roe"),
         ("quad-p3-o5", lambda: M.periodic_quad_2d(9, jitter=0.1), 3, 5, "HLLEP"),
         ("tet-p1-o2", None, 1, 2, "Roe"), ("tet-p1-o2-hllep", None, 1, 2, "HLLEP"), ("tet-p1-o4", None, 1, 4, "Roe"),
         ("tet-p1-o5", None, 1, 5, "HLLEP"), ("tet-p2-o4", None, 2, 4, "Roe"), ("tet-p2-o5", None, 2, 5, "HLLEP"),
         ("tet-p1-o2-m2", None, 1, 2, "Roe_M2"), ("tet-p3-o5", None, 3, 5, "Roe"),
         ("hex-p1-o3", lambda: M.tgv_mesh(5), 1, 3, "Roe"), ("hex-p1-o5", lambda: M.tgv_mesh(3), 1, 5, "HLLEP"),
         ("hex-p2-o5", lambda: M.tgv_mesh(5), 2, 5, "Roe")]


def _setup(mk, p, order, rs):
    import oracle
    from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction
    from tests.util import VR_HQM
    kw = dict(VR_HQM_PY, maxOrder=p, intOrder=order)
    es = dict(nVars=5, riemannSolverType=rs, muGas=0.0, ignoreVis=True)
    if mk is None:
        m = M.bump_channel_tet(5, 3, 2)
        o, far, types, vals, w = bump_oracle(m, p, rs, 0.0, 1, intOrder=order)
        vr = VariationalReconstruction(m, kw).construct(w)
        ev = EulerEvaluator(vr, es)
        ev.SetBC(types, vals)
        u0 = perturbed_state(m, far)
    else:
        m = mk()
        o = oracle.Oracle(m, dict(VR_HQM, maxOrder=p, intOrder=order),
                          dict(nVars=5, rsType=oracle.RS[rs], rsFixScale=1.0, rsIncFScale=1.0, gamma=1.4, Rgas=1.0, muGas=0.0, prGas=0.72,
                               TRef=273.15, CSutherland=110.4, muModel=0, ignoreVis=1))
        assert o.construct() == 0
        vr = VariationalReconstruction(m, kw).construct()
        ev = EulerEvaluator(vr, es)
        X = m.cell_coords().mean(1)
        X = 2 * np.pi * (X - X.min(0)) / np.maximum(np.ptp(X, axis=0), 1e-300)
        rho, vel, prs = 1 + 0.1 * np.sin(X[:, 0]), np.stack([0.6 + 0.1 * np.cos(X[:, 1]), 0.3 * np.sin(X[:, 0]), 0 * X[:, 0]], 1), 1 + 0.1 * np.cos(X[:, 1])
        u0 = np.concatenate([rho[:, None], rho[:, None] * vel, (prs / 0.4 + 0.5 * rho * (vel ** 2).sum(1))[:, None]], 1)
    rec0 = np.random.default_rng(3).normal(size=(m.n_cell, o.R, 5)) * 0.01 * np.abs(u0).mean(0)
    if m.cell_coords().shape[2] == 3 and m.dim == 2:
        rec0[:, :, 3] = 0
    u, rec = torch.tensor(u0, device="cuda"), torch.tensor(rec0, device="cuda")
    dt = torch.zeros(m.n_cell, dtype=torch.float64, device="cuda")
    ev.EvaluateDt(dt, u, 1.0)
    o.eval_dt(u0, 1.0)
    return m, o, ev, u0, rec0, u, rec


@pytest.mark.parametrize("name,mk,p,order,rs", CASES, ids=[c[0] for c in CASES])
def test_residual(name, mk, p, order, rs):
    m, o, ev, u0, rec0, u, rec = _setup(mk, p, order, rs)
    rhs = torch.full_like(u, 7.0)
    ev.EvaluateRHS(rhs, u, rec)
    # the bound of the residual's parity tests: FP64 sums of a few hundred terms
    assert relerr(rhs.cpu().numpy(), o.eval_rhs(u0, rec0)) < 1e-12


@pytest.mark.parametrize("name,mk,p,order,rs", CASES, ids=[c[0] for c in CASES])
def test_transpose(name, mk, p, order, rs):
    m, o, ev, u0, rec0, u, rec = _setup(mk, p, order, rs)
    g = torch.Generator(device="cuda").manual_seed(5)
    w, du, drec = (torch.randn(x.shape, dtype=torch.float64, device="cuda", generator=g) for x in (u, u, rec))
    a, b = ev.EvaluateRHSVJP(w, u, rec)
    t = ev.EvaluateRHSJVP(du, drec, u, rec)
    # two sums of the same products in another order: each entry carries some 1e3 rounded operations
    size = float((w * t).abs().sum() + (a * du).abs().sum() + (b * drec).abs().sum())
    assert abs(float((w * t).sum() - (a * du).sum() - (b * drec).sum())) < 1e3 * np.finfo(float).eps * size


@pytest.mark.parametrize("rs", ["Roe", "HLLEP"])
@pytest.mark.parametrize("p,order,n", [(3, 5, 47), (3, 5, 49), (3, 3, 47), (3, 3, 49), (2, 3, 68), (2, 3, 69)])
def test_transpose_on_both_sides_of_the_line_in_2d(p, order, n, rs):
    """The point-parallel kernel up to one wave of blocks (4,736 faces at degree 3, 9,472 at degree 2 with two points), the
    thread-per-face kernel beyond: <w, J v> = <J^T w, v> to the rounding of the sums."""
    from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction
    m = M.periodic_quad_2d(n, jitter=0.1)
    assert ((m.n_face + 31) // 32 > 148 * (4 - p)) == (n in (49, 69))
    vr = VariationalReconstruction(m, dict(VR_HQM_PY, maxOrder=p, intOrder=order)).construct()
    ev = EulerEvaluator(vr, dict(nVars=5, riemannSolverType=rs, muGas=0.0, ignoreVis=True))
    u = vr.BuildUDof(5)
    ev.InitializeUDOF(u, 2)
    g = torch.Generator("cuda").manual_seed(2)
    rand = lambda shape: torch.randn(shape, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
    rec = 0.01 * rand((m.n_cell, vr.R, 5)) * u.abs().mean(0)
    rec[:, :, 3] = 0
    ev.EvaluateDt(torch.zeros(m.n_cell, dtype=torch.float64, device="cuda"), u, 1.0)
    w, du, dr = rand(u.shape), rand(u.shape), rand(rec.shape)
    a, b = ev.EvaluateRHSVJP(w, u, rec)
    lhs = (w * ev.EvaluateRHSJVP(du, dr, u, rec)).flatten()
    rhs = torch.cat([(a * du).flatten(), (b * dr).flatten()])
    assert abs(float(lhs.sum() - rhs.sum())) < 1e-12 * float(lhs.abs().sum() + rhs.abs().sum())
