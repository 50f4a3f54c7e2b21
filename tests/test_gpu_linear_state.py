"""The native linear solve where its inputs are not finite and where one workspace serves several calls."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


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
