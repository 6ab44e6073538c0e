"""The one-launch CG solve of small 2D grids (pdg_cg2d.cu) against the oracle's
CG: fewer cells than SMs, more, every degree, the iteration cap, and a grid
that is too large for it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import pdg  # noqa: E402
import pdg_oracle as O  # noqa: E402


def solve(k, n, maxiter=5000, seed=3, react=False, f=None):
    import torch
    rng = np.random.default_rng(seed)
    nc = int(np.prod(n))
    K = np.exp(rng.standard_normal(nc))
    c = rng.uniform(0.5, 2.0, nc) if react else None
    bct = [1, 1, -1, 1, 1, 1]
    go = pdg.GridOperator(2, k, n, alpha=3.0, bctype=bct)
    P = O.Problem(2, k, n, alpha=3.0, bctype=bct, K=K, c=c)
    go.set_permeability(K)
    go.set_reaction(c)
    f = 1.0 + 0.1 * rng.standard_normal(nc) if f is None else f
    go.set_source(fc=f)
    P.set(fc=f)
    out = []
    for _ in range(2):
        ls = pdg.ISTLBackend_SEQ_MatrixFree_Base(go, maxiter=maxiter)
        u = torch.zeros(go.ndof, dtype=torch.float64, device="cuda")
        slp = pdg.StationaryLinearProblemSolver(go, ls, u, 1e-10)
        slp.apply()
        out.append((u.cpu().numpy(), slp.result().as_dict()))
    go.close()
    assert np.array_equal(out[0][0], out[1][0])   # the sums have a fixed order
    return out[0][0], out[0][1], P


@pytest.mark.parametrize("k", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [(1, 1), (7, 3), (17, 19)])
def test_against_oracle(k, n):
    u, res, P = solve(k, n, react=k == 3)
    ref, rres, _ = P.solve(solver="cg", op=0, reduction=1e-10)
    assert res["converged"]
    assert abs(res["iterations"] - rres.iterations) <= 1
    assert np.max(np.abs(u - ref)) <= 1e-8 * np.max(np.abs(ref))


def test_iteration_cap_and_zero_source():
    u, res, P = solve(2, (16, 16), maxiter=5)
    assert not res["converged"] and res["iterations"] == 5
    # the state of the recurrence after five iterations is the oracle's (the
    # residual norm itself need not fall: CG minimises the energy norm)
    ref, rres, _ = P.solve(solver="cg", op=0, reduction=1e-10, maxit=5)
    assert np.max(np.abs(u - ref)) <= 1e-8 * np.max(np.abs(ref))
    u, res, P = solve(2, (16, 16), f=np.zeros(256))
    assert res["converged"] and res["iterations"] == 0 and not u.any()


def test_large_grid_takes_the_launches_per_iteration():
    """400 x 400 cells of degree 2 do not fit the SMs' shared memory."""
    u, res, P = solve(2, (400, 400), maxiter=40)
    assert res["iterations"] == 40 and np.isfinite(u).all()
