"""Boundary-face kernels at the sizes where their blocks change shape: lists that fit one block of the wall-flux
reduction and lists that need several, every number of points per face (rows per block)."""
import numpy as np
import pytest
import torch

from dndsr_b200 import mesh as M
from tests.bump_case import bump_bc, bump_oracle, perturbed_state
from tests.util import VR_HQM, VR_HQM_PY, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(3, 2, 2), (4, 4, 6), (12, 6, 5)])  # 64, 256 and 648 boundary faces: one, one and three blocks
def test_wall_flux_is_the_sum_over_the_wall_faces(dims):
    from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction
    m = M.bump_channel_tet(*dims)
    far = M.freestream(0.8)
    types, vals, w = bump_bc(far)
    vr = VariationalReconstruction(m, dict(VR_HQM_PY, maxOrder=1, intOrder=2)).construct(w)
    ev = EulerEvaluator(vr, dict(nVars=5, riemannSolverType="Roe", muGas=0.0, ignoreVis=True))
    ev.SetBC(types, vals)
    u0, rec0 = perturbed_state(m, far, R=3)
    u, rec = torch.tensor(u0, device="cuda"), torch.tensor(rec0, device="cuda")
    dt = torch.zeros(m.n_cell, dtype=torch.float64, device="cuda")
    ev.EvaluateDt(dt, u, 1.0)
    ev.EvaluateRHS(torch.zeros_like(u), u, rec)
    ff = ev.get("faceFlux").reshape(-1, 5)[:m.n_face]
    walls = (m.face2cell[:, 1] < 0) & (types[m.face_zone] == 3)  # slip walls count without viscosity
    assert walls.sum() > 0
    # each of the n additions of the two orders rounds a partial sum of at most sum |f|
    bound = 2 * walls.sum() * np.finfo(float).eps * np.abs(ff[walls]).sum(0)
    assert np.all(np.abs(ev.get("fluxWallSum")[:5] + ff[walls].sum(0)) <= bound)


@pytest.mark.parametrize("p,intOrder", [(1, 2), (1, 4), (2, 5), (2, 6), (3, 6)])  # 3, 6, 7, 12, 12 points per face
def test_points_per_face_against_the_oracle(p, intOrder):
    """VR boundary term and boundary fluxes, the 1e-12 of the other parity tests; 64 boundary faces, so that the last
    block of 64 // points rows is ragged."""
    from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction
    m = M.renumber_by_color(M.bump_channel_tet(3, 2, 2))
    o, far, types, vals, w = bump_oracle(m, p, "Roe", 1e-3, 0, intOrder=intOrder, outflow_type=6, inflow_type=7, wall_type=2)
    vr = VariationalReconstruction(m, dict(VR_HQM_PY, maxOrder=p, intOrder=intOrder)).construct(w)
    ev = EulerEvaluator(vr, dict(nVars=5, riemannSolverType="Roe", muGas=1e-3, muModel=0, ignoreVis=False))
    ev.SetBC(types, vals)
    u0, rec0 = perturbed_state(m, far, R=o.R)
    u, rec = torch.tensor(u0, device="cuda"), torch.tensor(rec0, device="cuda")
    new, rhs, dt = torch.zeros_like(rec), torch.zeros_like(u), torch.zeros(m.n_cell, dtype=torch.float64, device="cuda")
    vr.DoReconstructionIter(rec, new, u, putIntoNew=True)
    assert relerr(new.cpu().numpy(), o.vr_iter(rec0, u0)) < 1e-12
    ev.EvaluateDt(dt, u, 5.0)
    o.eval_dt(u0, 5.0)
    ev.EvaluateRHS(rhs, u, rec)
    assert relerr(rhs.cpu().numpy(), o.eval_rhs(u0, rec0)) < 1e-12


@pytest.mark.parametrize("mk,nv,intOrder", [("tet", 5, 1), ("tet", 5, 0), ("hex", 5, 1), ("hex", 6, 1)])
def test_one_point_per_face_at_degree_3(mk, nv, intOrder):
    """The longest rows of the boundary reconstruction, R = 19, with the most rows to a block: VR boundary term against the
    oracle, and its transpose against the tangent."""
    import oracle
    from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction
    from tests.plate_case import plate_oracle, plate_perturbed
    if mk == "tet":
        m = M.renumber_by_color(M.bump_channel_tet(3, 2, 2))  # 64 boundary faces
        o, far, types, vals, w = bump_oracle(m, 3, "Roe", 0.0, 1, intOrder=intOrder)
        u0, rec0 = perturbed_state(m, far, R=o.R)
    else:
        m = M.renumber_by_color(M.flat_plate_hex(8, 6, 3, y1=1e-2, growth=1.3))
        o, far, mu, types, vals, w = plate_oracle(m, 3, "Roe", intOrder)
        u0, rec0 = plate_perturbed(m, far, R=o.R)
        if nv == 5:
            far, vals, u0, rec0 = far[:5], vals[:, :5].copy(), u0[:, :5].copy(), rec0[:, :, :5].copy()
            o = oracle.Oracle(m, dict(VR_HQM, maxOrder=3, intOrder=intOrder), dict(nVars=5, rsType=oracle.RS["Roe"], rsFixScale=1.0, rsIncFScale=1.0,
                              gamma=1.4, Rgas=1.0, muGas=0.0, prGas=0.72, TRef=273.15, CSutherland=110.4, muModel=0, ignoreVis=1))
            assert o.construct(w) == 0
            o.set_bc(types, vals)
    vr = VariationalReconstruction(m, dict(VR_HQM_PY, maxOrder=3, intOrder=intOrder)).construct(w)
    EulerEvaluator(vr, dict(nVars=nv, riemannSolverType="Roe", muGas=1e-3)).SetBC(types, vals)  # the sweep's boundary table too
    u, rec = torch.tensor(u0, device="cuda"), torch.tensor(rec0, device="cuda")
    new = torch.zeros_like(rec)
    vr.DoReconstructionIter(rec, new, u, putIntoNew=True)
    # both sides invert A in FP64: its condition number times a few roundings
    tol = 8 * np.finfo(float).eps * np.linalg.cond(o.get("matrixA").reshape(m.n_cell, o.R, o.R)).max()
    assert relerr(new.cpu().numpy(), o.vr_iter(rec0, u0)) < max(tol, 1e-12)
    if nv == 5:
        g = torch.Generator("cuda").manual_seed(1)
        cot, dRec, du = (torch.randn(t.shape, generator=g, dtype=torch.float64, device="cuda") for t in (rec, rec, u))
        vRec, vU = vr.DoReconstructionIterVJP(cot, rec, u)
        lhs = float((cot * vr.DoReconstructionIterJVP(dRec, du, rec, u)).sum())
        terms = torch.cat([(vRec * dRec).flatten(), (vU * du).flatten()])
        assert abs(lhs - float(terms.sum())) < 1e-12 * float(terms.abs().sum())
