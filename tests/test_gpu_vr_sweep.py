"""The VR Jacobi sweep's kernels on both sides of the layout rule, with ragged last tiles and warps and with boundary
faces, against the sweep written with the same coefficient arrays in torch (interior faces)."""
import numpy as np
import pytest
import torch

from dndsr_b200 import mesh as M
from tests.util import VR_HQM_PY

pytestmark = pytest.mark.gpu

CASES = [("tri-p1", lambda: M.periodic_quad_2d(7, jitter=0.1, split_tri=True), 1, 5), ("quad-p2", lambda: M.periodic_quad_2d(9, jitter=0.1), 2, 5),
         ("tri-p2", lambda: M.periodic_quad_2d(17, jitter=0.1, split_tri=True), 2, 5), ("quad-p3", lambda: M.periodic_quad_2d(11, jitter=0.1), 3, 5),
         ("tri-p3-tiled", lambda: M.periodic_quad_2d(101, jitter=0.1, split_tri=True), 3, 5),  # 20,402 cells: the last tile has 18
         ("tet-p1", lambda: M.bump_channel_tet(5, 3, 2), 1, 5), ("tet-p2", lambda: M.bump_channel_tet(5, 3, 2), 2, 5),
         ("tet-p2-tiled", lambda: M.bump_channel_tet(41, 21, 4), 2, 5),  # 20,664 cells, 24 in the last tile
         ("hex-p1", lambda: M.tgv_mesh(5), 1, 5), ("hex-p2", lambda: M.tgv_mesh(7), 2, 5), ("hex-p2-tiled", lambda: M.tgv_mesh(29), 2, 5),
         ("hex-p1-sa", lambda: M.tgv_mesh(7), 1, 6), ("tet-p1-sa", lambda: M.bump_channel_tet(5, 3, 2), 1, 6)]


@pytest.mark.parametrize("name,mk,p,nv", CASES, ids=[c[0] for c in CASES])
def test_sweep(name, mk, p, nv):
    from dndsr_b200.solver import VariationalReconstruction
    m = mk()
    bnd = m.face2cell[:, 1] < 0
    n_zone = int(m.face_zone.max()) + 1
    vr = VariationalReconstruction(m, dict(VR_HQM_PY, maxOrder=p, intOrder=5, jacobiRelax=0.7))
    # weights of zero take the boundary term out of the sweep, so that the interior faces are what is compared
    vr.construct(np.where(np.arange(n_zone)[:, None] > 0, 0.0, 1.0) * np.ones((n_zone, 4)) if bnd.any() else None)
    if bnd.any():
        vr._c.SetBoundary(np.where(np.arange(n_zone) > 0, 9, 0).astype(np.int32), np.zeros((n_zone, nv)), nv, 1.4, 1.0)
    nf, R, nc = m.cell2face.shape[1], vr.R, m.n_cell
    g = torch.Generator(device="cuda").manual_seed(3)
    uRec = torch.randn((nc, R, nv), dtype=torch.float64, device="cuda", generator=g)
    u = torch.randn((nc, nv), dtype=torch.float64, device="cuda", generator=g)
    side = m.face2cell[m.cell2face, 0] == np.arange(nc)[:, None]
    nbr = torch.as_tensor(np.where(side, m.face2cell[m.cell2face, 1], m.face2cell[m.cell2face, 0]), device="cuda")
    mat = torch.as_tensor(vr.get("matrixAAInvB").reshape(nc, nf + 1, R, R)[:, 1:], device="cuda") * (nbr >= 0)[:, :, None, None]
    vec = torch.as_tensor(vr.get("vectorAInvB").reshape(nc, nf, R), device="cuda") * (nbr >= 0)[:, :, None]
    o = nbr.clamp_min(0)
    const = torch.einsum("cfi,cfv->civ", vec, u[o] - u[:, None])
    full = torch.einsum("cfij,cfjv->civ", mat, uRec[o]) + const
    new = torch.empty_like(uRec)
    # each entry sums nf (R + 1) products; the entries are of order one times the row sums of the coefficients
    size = float(torch.einsum("cfij->ci", mat.abs()).max() + vec.abs().sum(1).max()) * 6
    bound = nf * (R + 1) * np.finfo(float).eps * size
    for kw, ref in ((dict(), 0.3 * uRec + 0.7 * full), (dict(recordInc=True), uRec - full), (dict(recordInc=True, uRecIsZero=True), -const)):
        new.fill_(7.0)
        vr.DoReconstructionIter(uRec, new, u, putIntoNew=True, **kw)
        assert float((new - ref).abs().max()) < bound, kw
    vr.DoReconstructionIter(uRec, new, u, putIntoNew=True, precision="fp32")  # coefficients rounded to 24 bits
    assert float((new - (0.3 * uRec + 0.7 * full)).abs().max()) < 2 ** -24 * size
