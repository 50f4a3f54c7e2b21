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


def _bump(nx=6, ny=4, nz=2):
    from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction
    far = M.freestream(0.8)
    types, vals, w = bump_bc(far)
    vr = VariationalReconstruction(M.bump_channel_tet(nx, ny, nz), dict(VR_HQM_PY, maxOrder=1, intOrder=2)).construct(w)
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


@pytest.mark.parametrize("linear", [dict(), dict(gmresCode=1, nGmresSpace=5), dict(gmresCode=2, nGmresSpace=5)])
def test_nonphysical_state_is_reported(linear):
    """The native iteration and the closures report the same error, and neither leaves any of it behind: with the state
    restored the same solver runs as a new one does (90 cells: a vector of 450 elements ends within a group of four)."""
    from dndsr_b200.capi import DndsbError

    def solver(cls):
        vr, ev, u = _bump(5, 3, 1)
        s = cls(vr, ev, I.SolverConfig(odeCode=1, dtImplicit=1e100, nTimeStep=1, nTimeStepInternal=3, CFL=5.0, **linear))
        assert vr.mesh.n_cell % 4 != 0 and s._native() == (cls is I.ImplicitSolver)
        return s, u

    errors = []
    for cls in (I.ImplicitSolver, Closures):
        s, u = solver(cls)
        good = u.clone()
        u[5, 0] = -1.0
        with pytest.raises(DndsbError) as e:
            s.run(u)
        code, text = str(e.value).split(":")[0], str(e.value).split(":")[-1]
        errors.append((e.value.code, code, text))
        u.copy_(good)
        for t in (s.uRec, s.uRecNew):
            t.zero_()
        s.CFLNow, s.resBase = s.cfg.CFL, None
        s.cfg.res_history.clear()
        s.run(u)
        fresh, v = solver(cls)
        fresh.run(v)
        assert bool(torch.isfinite(u).all()) and not torch.equal(u, good)
        assert torch.equal(u, v) and torch.equal(s.uRec, fresh.uRec) and s.cfg.res_history == fresh.cfg.res_history
    assert errors[0] == errors[1]
