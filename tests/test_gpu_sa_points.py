"""The SA source and its reverse over the numbers of points per cell and face (rows per block of their kernels), with
the SA variable negative in some cells: the source against the oracle, the VJP against the forward-mode JVP."""
import numpy as np
import pytest
import torch

from dndsr_b200 import mesh as M
from tests.plate_case import plate_oracle, plate_perturbed
from tests.util import VR_HQM_PY, relerr

pytestmark = pytest.mark.gpu


# 8, 27, 64 points per cell (4, 9, 16 per face)
@pytest.mark.parametrize("p,intOrder", [(1, 3), (1, 5), (1, 6), (2, 5), (2, 6)])
@pytest.mark.parametrize("muModel", [0, 1])
def test_source_and_reverse(p, intOrder, muModel):
    from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction
    m = M.renumber_by_color(M.flat_plate_hex(7, 6, 3, y1=1e-3, growth=1.8))  # 126 cells: a ragged last block
    o, far, mu, types, vals, w = plate_oracle(m, p, intOrder=intOrder)
    vr = VariationalReconstruction(m, dict(VR_HQM_PY, maxOrder=p, intOrder=intOrder)).construct(w)
    # Sutherland with TRef at the free-stream temperature: mu varies with the state
    ev = EulerEvaluator(vr, dict(nVars=6, riemannSolverType="Roe", muGas=mu, muModel=muModel, prGas=0.72, TRef=1.0, CSutherland=0.4))
    ev.SetBC(types, vals)
    ev.SetWallDistance(M.plate_wall_distance(vr.get("cellPP").reshape(m.n_cell, -1, 3)))
    u0, rec0 = plate_perturbed(m, far, R=o.R)
    u0[::7, 5] *= -0.5
    u, rec = torch.tensor(u0, device="cuda"), torch.tensor(rec0, device="cuda")
    dt, rhs = torch.zeros(m.n_cell, dtype=torch.float64, device="cuda"), torch.zeros_like(u)
    ev.EvaluateDt(dt, u, 1.0)
    ev.EvaluateRHS(rhs, u, rec)
    if muModel == 0:  # the oracle of this set-up has constant viscosity
        o.eval_dt(u0, 1.0)
        ref = o.eval_rhs(u0, rec0)
        assert relerr(rhs.cpu().numpy(), ref) < 1e-12
        assert relerr(rhs.cpu().numpy()[:, 5], ref[:, 5]) < 1e-12
    g = torch.Generator(device="cuda").manual_seed(2)
    for v in (range(6), [5]):  # all variables, then the SA equation alone (its source is not drowned by the fluxes)
        wt = torch.zeros_like(u)
        wt[:, list(v)] = torch.randn((m.n_cell, len(list(v))), dtype=torch.float64, device="cuda", generator=g)
        wt[:, list(v)] *= torch.as_tensor(vr.get("volume"), device="cuda")[:, None]
        du, dr = torch.randn(u.shape, dtype=torch.float64, device="cuda", generator=g), torch.randn(rec.shape, dtype=torch.float64, device="cuda", generator=g)
        gu, gr = ev.EvaluateRHSVJP(wt, u, rec)
        jv = ev.EvaluateRHSJVP(du, dr, u, rec)
        a, b = wt * jv, torch.cat([(gu * du).ravel(), (gr * dr).ravel()])
        # both sums round in the size of their terms
        assert abs(float(a.sum() - b.sum())) < 1e-12 * float(a.abs().sum() + b.abs().sum())
