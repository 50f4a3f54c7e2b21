"""The native linear solve where its inputs are not finite and where one workspace serves several calls."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _box(n=7):
    """n^2 quadrilaterals, 5 n^2 unknowns: with n odd a vector ends within a group of four."""
    from dndsr_b200 import mesh as M
    from dndsr_b200.solver import EulerEvaluator, VariationalReconstruction
    from tests.util import VR_HQM_PY
    vr = VariationalReconstruction(M.periodic_quad_2d(n, jitter=0.1), dict(VR_HQM_PY, maxOrder=1)).construct()
    ev = EulerEvaluator(vr, dict(nVars=5, riemannSolverType="Roe", muGas=0.0, ignoreVis=True))
    u = vr.BuildUDof(5)
    ev.InitializeUDOF(u, 2)
    dTau = torch.zeros(vr.mesh.n_cell, dtype=torch.float64, device="cuda")
    ev.EvaluateDt(dTau, u, 5.0)
    return ev, u, dTau, torch.tensor(np.random.default_rng(5).normal(size=(vr.mesh.n_cell, 5)), device="cuda")


def _solve(ev, u, dTau, rhs, **kw):
    x = torch.zeros_like(rhs)
    ev.SolveLinear(0.5, dTau, 0.1, u, rhs, x, **kw)
    return x


def _least_squares(H, beta, k):
    """min |beta e1 - H y| by Givens rotations in the order of the device's chain; H[j] is column j."""
    dmax = lambda a, b: a if a > b else b  # noqa: E731  the device's maximum, which is not symmetric in a NaN
    R = np.zeros((k + 1, k))
    for j in range(k):
        R[:min(j + 2, k + 1), j] = H[j, :min(j + 2, k + 1)]
    g = np.zeros(k + 1)
    g[0] = beta
    for j in range(k):
        a, b = R[j, j], R[j + 1, j]
        r = np.sqrt(a * a + b * b)
        c, s = (a / r, b / r) if r > 0 else (1.0, 0.0)
        x0, x1 = R[j, j:].copy(), R[j + 1, j:].copy()
        R[j, j:], R[j + 1, j:] = c * x0 + s * x1, -s * x0 + c * x1
        g[j], g[j + 1] = c * g[j] + s * g[j + 1], -s * g[j] + c * g[j + 1]
    rmax = 0.0
    for j in range(k):
        rmax = dmax(rmax, abs(R[j, j]))
    y = np.zeros(k)
    for j in range(k - 1, -1, -1):
        if abs(R[j, j]) > 1e-14 * rmax:
            y[j] = (g[j] - sum(R[j, l] * y[l] for l in range(j + 1, k))) / R[j, j]
    return y


@pytest.mark.parametrize("k,at", [(1, None), (5, None), (5, (0, 0)), (5, (1, 1)), (5, (3, 2)), (32, None), (32, (1, 1)), (32, (3, 30))])
def test_least_squares_with_an_infinite_entry(k, at):
    """Every lane of the least squares' warp decides alike, also where the largest diagonal is not a number."""
    from dndsr_b200.solver import _C
    C = _C()
    n, f64 = 8, dict(dtype=torch.float64, device="cuda")
    rng = np.random.default_rng(3)
    H = np.triu(rng.normal(size=(k, k + 1)).T, -1).T  # column j in row j, upper Hessenberg
    H[np.arange(k), np.arange(k)] += 3.0
    H[k - 1] = 0  # arnoldi writes the last column: zero products against the empty columns, then the norm
    if at is not None:
        H[at[1], at[0]] = np.inf
    V = torch.zeros((k + 1, C.krylov_ld(n)), **f64)
    V[k, :n] = 1.0
    Hd = torch.tensor(H.reshape(-1), **f64)
    gsc, cs, work = torch.zeros(8 + k, **f64), torch.ones(k + 1, **f64), torch.zeros(C.krylov_work_bytes(), dtype=torch.uint8, device="cuda")
    r = torch.zeros(n, **f64)
    r[0] = 2.0
    V0 = V.clone()
    C.krylov_start(r, V, gsc, cs, work, k)  # beta = 2 and the work area's weights
    V.copy_(V0)
    cs.fill_(1.0)
    res = torch.zeros(1, **f64)
    C.krylov_arnoldi(n, k - 1, k, V, Hd, cs, gsc, res, work)
    H[k - 1, k] = np.sqrt(n)
    with np.errstate(invalid="ignore"):
        y = _least_squares(H, 2.0, k)
    got = gsc[8:8 + k].cpu().numpy()
    # a chain of k rotations and substitutions of a matrix of condition below 1e3
    assert np.allclose(got, y, rtol=1e-10, atol=1e-12, equal_nan=True), (got, y)


DIRECT, SWEEPS, GMRES = dict(gmresCode=0), dict(gmresCode=0, sgsIter=8), dict(gmresCode=1, nGmresSpace=6)


@pytest.mark.parametrize("first,second", [(DIRECT, DIRECT), (DIRECT, GMRES), (GMRES, DIRECT), (DIRECT, SWEEPS), (GMRES, GMRES)])
def test_solves_on_two_streams_follow_each_other(first, second):
    """Two callers' streams, one workspace: the second solve waits until the first is done (held back here by other work
    on its stream), and both give what they give in turn."""
    ev, u, dTau, rhs = _box(41)
    rhs2 = torch.flip(rhs, [0]) * 2
    want = [_solve(ev, u, dTau, r, **k).clone() for r, k in ((rhs, first), (rhs2, second))]
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    big = torch.ones((4096, 4096), device="cuda")
    x1, x2, held = torch.zeros_like(rhs), torch.zeros_like(rhs), torch.empty_like(big)
    torch.cuda.synchronize()
    for _ in range(3):
        done1 = torch.cuda.Event()
        x1.zero_(), x2.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(s1):
            for _ in range(20):
                torch.mm(big, big, out=held)
            ev.SolveLinear(0.5, dTau, 0.1, u, rhs, x1, **first)
            done1.record()
        with torch.cuda.stream(s2):
            ev.SolveLinear(0.5, dTau, 0.1, u, rhs2, x2, **second)
        s2.synchronize()
        assert done1.query()
        torch.cuda.synchronize()
        assert torch.equal(x1, want[0]) and torch.equal(x2, want[1])


def test_solve_on_two_streams_of_a_capture():
    """The same order inside a captured graph; solves before and after it, and its replay, give the same."""
    ev, u, dTau, rhs = _box(41)
    want = _solve(ev, u, dTau, rhs).clone()
    x1, x2 = torch.zeros_like(rhs), torch.zeros_like(rhs)
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        side.wait_stream(torch.cuda.current_stream())
        ev.SolveLinear(0.5, dTau, 0.1, u, rhs, x1)
        with torch.cuda.stream(side):
            ev.SolveLinear(0.5, dTau, 0.1, u, rhs, x2)
        torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(_solve(ev, u, dTau, rhs), want)  # outside the capture again
    torch.cuda.synchronize()
    for _ in range(2):
        x1.zero_(), x2.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(x1, want) and torch.equal(x2, want)


@pytest.mark.parametrize("other", [dict(nGmresSpace=5), dict(nGmresSpace=10, sgsIter=1), dict(nGmresSpace=10, nGmresIter=2),
                                   dict(nGmresSpace=10, jacobiCode=0), dict(nGmresSpace=10, gmresCode=2)])
def test_recorded_sequence_is_of_its_settings(other):
    """A solve that records nothing between two that do: the third replays the second's settings, not the first's."""
    ev, u, dTau, rhs = _box()
    first, other = dict(gmresCode=1, nGmresSpace=10), dict(dict(gmresCode=1), **other)
    a = _solve(ev, u, dTau, rhs, useGraph=True, **first)
    b = _solve(ev, u, dTau, rhs, useGraph=False, **other)
    c = _solve(ev, u, dTau, rhs, useGraph=True, **other)
    assert not torch.equal(a, b)
    assert torch.equal(b, c)
    assert torch.equal(a, _solve(ev, u, dTau, rhs, useGraph=True, **first))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("gmresCode", [1, 2])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_solve_after_a_nonfinite_one(bad, gmresCode, precision):
    """Nothing of a solve that is not finite stays in the workspace, the Krylov columns' ends included."""
    kw = dict(gmresCode=gmresCode, nGmresSpace=6, precision=precision)
    ev, u, dTau, rhs = _box()
    poisoned = rhs.clone()
    poisoned[3, 1] = bad
    _solve(ev, u, dTau, poisoned, **kw)
    x = _solve(ev, u, dTau, rhs, **kw)
    fresh = _box()[0]
    fresh.EvaluateDt(torch.zeros_like(dTau), u, 5.0)
    assert bool(torch.isfinite(x).all()) and float(x.abs().max()) > 0
    assert torch.equal(x, _solve(fresh, u, dTau, rhs, **kw))
