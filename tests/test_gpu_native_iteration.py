"""The native pseudo-iteration of ImplicitSolver against its closures (a subclass that overrides one keeps them): the same
states up to rounding, the same history length, the same error."""
import numpy as np
import pytest
import torch

from dndsr_b200 import implicit as I
from dndsr_b200 import mesh as M
from tests.bump_case import bump_bc
from tests.plate_case import plate_bc, plate_perturbed, plate_state
from tests.util import VR_HQM_PY

pytestmark = pytest.mark.gpu


class Closures(I.ImplicitSolver):
    def fincrement(self, cx, cxInc, alpha):
        super().fincrement(cx, cxInc, alpha)


def _vortex():
    from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction
    vr = VariationalReconstruction(M.iv_mesh(11), dict(VR_HQM_PY, maxOrder=2)).construct()
    ev = EulerEvaluator(vr, dict(nVars=5, riemannSolverType="Roe", muGas=0.0, ignoreVis=True))
    u = vr.BuildUDof(5)
    ev.InitializeUDOF(u, 2)
    return vr, ev, u


def _bump():
    from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction
    far = M.freestream(0.8)
    types, vals, w = bump_bc(far)
    vr = VariationalReconstruction(M.bump_channel_tet(6, 4, 2), dict(VR_HQM_PY, maxOrder=1, intOrder=2)).construct(w)
    ev = EulerEvaluator(vr, dict(nVars=5, riemannSolverType="Roe_M2", muGas=0.0, ignoreVis=True))
    ev.SetBC(types, vals)
    u = vr.BuildUDof(5)
    u[:] = torch.tensor(far, device="cuda")
    return vr, ev, u


def _plate():
    from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction
    m = M.flat_plate_hex(8, 6, 3, y1=1e-3, growth=1.6)
    far, mu = plate_state()
    types, vals, w = plate_bc(far)
    vr = VariationalReconstruction(m, dict(VR_HQM_PY, maxOrder=1, intOrder=3)).construct(w)
    ev = EulerEvaluator(vr, dict(nVars=6, riemannSolverType="Roe", muGas=mu, muModel=0, prGas=0.72))
    ev.SetBC(types, vals)
    ev.SetWallDistance(M.plate_wall_distance(vr.get("cellPP").reshape(m.n_cell, -1, 3)))
    return vr, ev, torch.tensor(plate_perturbed(m, far), device="cuda")


@pytest.mark.parametrize("mk,cfg", [(_vortex, dict(odeCode=0, nTimeStep=2, nTimeStepInternal=6, CFL=50.0)),
                                    (_vortex, dict(odeCode=101, nTimeStep=2, nTimeStepInternal=6, CFL=50.0, gmresCode=1, nGmresSpace=5,
                                                   normOrd=2, useVolWiseResidual=True, nInternalRecStep=2)),
                                    (_bump, dict(odeCode=1, dtImplicit=1e100, nTimeStep=1, nTimeStepInternal=8, CFL=20.0, sgsIter=1, normOrd=3)),
                                    (_plate, dict(odeCode=1, dtImplicit=1e100, nTimeStep=1, nTimeStepInternal=6, CFL=5.0))])
def test_states_agree(mk, cfg):
    out = []
    for cls in (I.ImplicitSolver, Closures):
        vr, ev, u = mk()
        c = I.SolverConfig(**dict(dict(dtImplicit=0.02, rhsThresholdInternal=0.0), **cfg))
        s = cls(vr, ev, c)
        assert s._native() == (cls is I.ImplicitSolver)
        s.run(u)
        out.append((u, s.uRec.clone(), c.res_history, s.n_rhs))
    (a, ra, ha, na), (b, rb, hb, nb) = out
    assert len(ha) == len(hb) and na == nb
    # the residual and the update round once more or less per iteration; a few dozen iterations near a steady state
    assert float((a - b).abs().max() / b.abs().max()) < 1e-13
    assert float((ra - rb).abs().max() / rb.abs().max()) < 1e-12
    assert np.allclose([h[2] for h in ha], [h[2] for h in hb], rtol=1e-8)


def test_nonphysical_state_is_reported():
    from dndsr_b200.capi import DndsbError
    vr, ev, u = _bump()
    u[5, 0] = -1.0
    s = I.ImplicitSolver(vr, ev, I.SolverConfig(odeCode=1, dtImplicit=1e100, nTimeStep=1, nTimeStepInternal=3, CFL=5.0))
    assert s._native()
    with pytest.raises(DndsbError):
        s.run(u)
